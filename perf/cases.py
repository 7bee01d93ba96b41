"""The work a user of cortexsdr_b200 has it do, as cases that can be timed and checked.

Each case goes through the public entry points: products of activations with compressed weights
(`Segment.matmul_device`, `matmul_group_device`, `matmul_queue_device`), reconstruction
(`Segment.decompress_device`), encoding (`HierarchicalSDRStrategy.compress`) and decoder passes
over an archive (`Decoder.step`, `Decoder.forward`). Weights are synthetic payloads of the
reference's format: a Gaussian dictionary and uniformly random (atom, sign) codes, scaled so that
the weights have standard deviation 0.02 - decoding costs the same whichever atoms codes name.
"""
import math
import os
import struct
import tempfile

import numpy as np
import torch

import cortexsdr_b200 as cs

STAGES, DECAY, WEIGHT_STD = 3, 0.5, 0.02

# Block shapes of the two decoders the benchmark runs, and the vocabulary of each.
SHAPES = {
    "llama7b": dict(hidden=4096, q_heads=32, kv_heads=32, head_dim=128, inter=11008, vocab=32000, kv_atoms=512, eps=1e-5),
    "qwen0.5b": dict(hidden=896, q_heads=14, kv_heads=2, head_dim=64, inter=4864, vocab=151936, kv_atoms=128, eps=1e-6),
}
ROPE_THETA = 1e6


def _product(name, rows, cols, batch, dtype="f32", tile=0, atoms=512, k=8, layout="feature", members=1):
    kind = "product" if members == 1 else "group"
    return dict(name=name, kind=kind, rows=rows, cols=cols, batch=batch, dtype=dtype, tile=tile, atoms=atoms, k=k,
                layout=layout, members=members)


def listed():
    return [
        # the smallest call: one query projection of a 0.5B-class decoder for one token
        _product("one_896x896_m1", 896, 896, 1),
        # the products of one token that share an activation: gate and up of a 0.5B-class MLP
        _product("pair_4864x896_m1", 4864, 896, 1, members=2),
        # a whole pass of independent one-token products, together larger than the L2 cache: the
        # library's headline workload
        dict(name="list_32x11008x4096_m1", kind="list", rows=11008, cols=4096, batch=1, dtype="f32", tile=0, atoms=512, k=8,
             layout="feature", members=32),
        # a few concurrent users decoding: the MLP projection for eight tokens
        _product("one_11008x4096_m8", 11008, 4096, 8, "bf16", layout="token"),
        # a short prompt, or 64 users: the MLP's way back
        _product("one_4096x11008_m64", 4096, 11008, 64, "bf16", layout="token"),
        # a prompt of 512 tokens
        _product("one_11008x4096_m512", 11008, 4096, 512, "bf16", layout="token"),
        # weights encoded as 128x128 tiles (the encoder's default geometry): one token
        _product("tiles_4096x4096_m1", 4096, 4096, 1, tile=128),
        # and a prompt of 128 tokens against the widest MLP of the benchmark
        _product("tiles_14336x4096_m128", 14336, 4096, 128, "bf16", tile=128, layout="token"),
        # a weight taken out of its archive as a matrix, with ragged edges on both sides
        dict(name="decompress_4099x4101", kind="decompress", rows=4099, cols=4101, tile=128, atoms=512, k=8),
        # a square projection put into an archive: host matrix in, payload out
        dict(name="encode_4096x4096", kind="encode", rows=4096, cols=4096, atoms=512, k=8),
        # serving: sixteen sequences at context 1024, four given tokens each (blocks of the
        # 7B-class decoder at full width, embedding and head included)
        dict(name="step_7b_b16_ctx1024", kind="step", shape="llama7b", layers=4, batch=16, context=1024, steps=4),
        # a prompt of 1024 tokens through blocks of the same decoder
        dict(name="prompt_7b_1024", kind="prompt", shape="llama7b", layers=2, tokens=1024, steps=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["product", "tiles", "group", "list", "decompress", "encode", "step", "prompt"],
                       [34, 16, 10, 8, 8, 4, 10, 10])[0]
    if kind in ("step", "prompt"):
        shape = rng.choice(sorted(SHAPES))
        if kind == "step":
            return dict(kind=kind, shape=shape, layers=rng.randint(2, 4), batch=rng.randint(1, 16), context=_log(rng, 33, 1024),
                        steps=rng.randint(2, 4))
        return dict(kind=kind, shape=shape, layers=2, tokens=_log(rng, 17, 1024), steps=0)
    if kind == "encode":
        return dict(kind=kind, rows=_log(rng, 1024, 4096), cols=4 * _log(rng, 128, 1024), atoms=rng.choice([128, 256, 512]), k=rng.choice([5, 8]))
    if kind == "decompress":
        tile = rng.choice([0, 16, 32, 64, 128])
        return dict(kind=kind, rows=_log(rng, 512, 4096), cols=_log(rng, 512, 4096), tile=tile, atoms=rng.choice([256, 512]), k=rng.choice([5, 8]))
    # widths are multiples of 4 three times in four; the rest are what they are
    rows = _log(rng, 300, 14336)
    cols = 4 * _log(rng, 64, 2752) if rng.random() < 0.75 else _log(rng, 257, 11008)
    atoms, k = rng.choice([128, 256, 300, 512]), rng.choice([4, 5, 8])
    dtype, layout = rng.choice(["f32", "bf16"]), rng.choice(["feature", "token"])
    if kind == "group":
        return dict(kind=kind, rows=rows, cols=cols, batch=_log(rng, 1, 16), dtype=dtype, tile=0, atoms=atoms, k=k, layout=layout,
                    members=rng.randint(2, 3))
    if kind == "list":
        return dict(kind=kind, rows=min(rows, 11008), cols=min(cols, 4096), batch=_log(rng, 1, 4), dtype="f32", tile=0, atoms=512, k=8,
                    layout="feature", members=rng.randint(5, 16))
    tile = rng.choice([16, 32, 64, 128]) if kind == "tiles" else 0
    if tile:
        rows, cols = min(rows, 11008), min(cols, 8192)
    return dict(kind="product", rows=rows, cols=cols, batch=_log(rng, 1, 512), dtype=dtype, tile=tile, atoms=atoms, k=k, layout=layout, members=1)


# ---- payloads ----

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _scales():
    return [DECAY ** s for s in range(STAGES)]


def _parts(gen, rows, cols, tile, atoms, k):
    """(dictionary [K][Tr*Tc] fp32, codes [tiles][S*k] uint16 as int32, edge floats) on the GPU."""
    tr, tc = (tile, tile) if tile else (1, cols)
    rf, cf = rows // tr * tr, cols // tc * tc
    n_tiles = (rf // tr) * (cf // tc)
    std = WEIGHT_STD / math.sqrt(k * sum(s * s for s in _scales()))
    dictionary = torch.randn(atoms, tr * tc, generator=gen, device="cuda") * std
    codes = torch.randint(0, atoms, (n_tiles, STAGES * k), generator=gen, device="cuda", dtype=torch.int32)
    codes |= torch.randint(0, 2, codes.shape, generator=gen, device="cuda", dtype=torch.int32) << 15
    edges = torch.randn(rf * (cols - cf) + (rows - rf) * cols, generator=gen, device="cuda") * WEIGHT_STD
    return dictionary, codes, edges


def _payload(parts, rows, cols, tile, k):
    dictionary, codes, edges = parts
    tr, tc = (tile, tile) if tile else (1, cols)
    head = struct.pack("<4sIIIIHHHBBfI", b"HSDR", 2, rows, cols, codes.shape[0], tr, tc, dictionary.shape[0], STAGES, k, DECAY,
                       4 * edges.numel())
    body = (np.frombuffer(head, np.uint8), np.array(_scales(), np.float32).view(np.uint8), dictionary.cpu().numpy().view(np.uint8).reshape(-1),
            codes.cpu().numpy().astype(np.uint16).view(np.uint8).reshape(-1), edges.cpu().numpy().view(np.uint8))
    return np.concatenate(body)


def _payload_bytes(rows, cols, tile, atoms, k):
    tr, tc = (tile, tile) if tile else (1, cols)
    rf, cf = rows // tr * tr, cols // tc * tc
    tiles = (rf // tr) * (cf // tc)
    return 40 + 4 * STAGES + 4 * atoms * tr * tc + 2 * tiles * STAGES * k + 4 * (rf * (cols - cf) + (rows - rf) * cols)


def _dense(parts, rows, cols, tile, k):
    """The weight in 64 bits."""
    dictionary, codes, edges = (p.double() if p.is_floating_point() else p.long() for p in parts)
    tr, tc = (tile, tile) if tile else (1, cols)
    out = torch.zeros(codes.shape[0], tr * tc, dtype=torch.float64, device="cuda")
    for s in range(codes.shape[1]):
        c = codes[:, s]
        out += dictionary[c & 0x7FFF] * ((1 - 2 * (c >> 15)) * _scales()[s // k]).double()[:, None]
    rf, cf = rows // tr * tr, cols // tc * tc
    w = torch.empty(rows, cols, dtype=torch.float64, device="cuda")
    w[:rf, :cf] = out.view(rf // tr, cf // tc, tr, tc).permute(0, 2, 1, 3).reshape(rf, cf)
    n = rf * (cols - cf)
    w[:rf, cf:] = edges[:n].view(rf, cols - cf)
    w[rf:] = edges[n:].view(rows - rf, cols)
    return w


# ---- products ----

def _activations(gen, case):
    """[batch][cols] in the case's layout and type, N(0, 1) as normalised activations are."""
    shape = (case["batch"], case["cols"]) if case["layout"] == "token" else (case["cols"], case["batch"])
    x = torch.randn(shape, generator=gen, device="cuda")
    return x.bfloat16() if case["dtype"] == "bf16" else x


def _product_inputs(case, seed):
    """Generators give the same parts to prepare() and exact()."""
    gen = _generator(seed)
    for _ in range(case["members"]):
        yield _parts(gen, case["rows"], case["cols"], case["tile"], case["atoms"], case["k"])
    for _ in range(case["members"] if case["kind"] == "list" else 1):
        yield _activations(gen, case)


def _prepare_product(case, seed):
    n, segs, xs = case["members"], [], []
    for i, p in enumerate(_product_inputs(case, seed)):
        if i < n:
            segs.append(cs.Segment.from_payload(_payload(p, case["rows"], case["cols"], case["tile"], case["k"])))
        else:
            xs.append(p)
    shape = (case["batch"], case["rows"]) if case["layout"] == "token" else (case["rows"], case["batch"])
    ys = [torch.empty(shape, device="cuda") for _ in range(n)]
    dtype = cs.DTYPE_BF16 if case["dtype"] == "bf16" else cs.DTYPE_F32
    layout = cs.TOKEN_MAJOR if case["layout"] == "token" else cs.FEATURE_MAJOR
    torch.cuda.synchronize()
    state = dict(kind=case["kind"], segs=segs, xs=xs, ys=ys, dtype=dtype, layout=layout, batch=case["batch"])
    if case["kind"] == "list":
        state["tasks"] = [(s, x.data_ptr(), dtype, layout, case["batch"], y.data_ptr(), layout) for s, x, y in zip(segs, xs, ys)]
        state["prepared"] = None
    return state


def _run_product(s):
    if s["kind"] == "product":
        s["segs"][0].matmul_device(s["xs"][0].data_ptr(), s["dtype"], s["layout"], s["batch"], s["ys"][0].data_ptr(), s["layout"])
    elif s["kind"] == "group":
        cs.Segment.matmul_group_device(s["segs"], s["xs"][0].data_ptr(), s["dtype"], s["layout"], s["batch"],
                                       [y.data_ptr() for y in s["ys"]], s["layout"])
    else:
        s["prepared"] = cs.Segment.matmul_queue_device(s["tasks"], s["prepared"])
    return s["ys"]


def _exact_product(case, seed):
    parts = list(_product_inputs(case, seed))
    n, out = case["members"], []
    for i in range(n):
        x = parts[n + (i if case["kind"] == "list" else 0)].double()
        w = _dense(parts[i], case["rows"], case["cols"], case["tile"], case["k"])
        out.append(x @ w.T if case["layout"] == "token" else w @ x)
        del w
    return out


# ---- decoder ----

def _linears(spec, layers):
    """(name, rows, cols, atoms, segment type, layer) of every compressed tensor, in file order."""
    h, qd, kd = spec["hidden"], spec["q_heads"] * spec["head_dim"], spec["kv_heads"] * spec["head_dim"]
    out = [("token_embd.weight", spec["vocab"], h, 512, 13, 0)]
    for i in range(layers):
        p = "blk.%d." % i
        out += [(p + "attn_q.weight", qd, h, 512, 11, i), (p + "attn_k.weight", kd, h, spec["kv_atoms"], 11, i),
                (p + "attn_v.weight", kd, h, spec["kv_atoms"], 11, i), (p + "attn_output.weight", h, qd, 512, 11, i),
                (p + "ffn_gate.weight", spec["inter"], h, 512, 12, i), (p + "ffn_up.weight", spec["inter"], h, 512, 12, i),
                (p + "ffn_down.weight", h, spec["inter"], 512, 12, i)]
    return out + [("output.weight", spec["vocab"], h, 512, 13, 0)]


def _decoder_parts(case, seed):
    gen = _generator(seed)
    for name, rows, cols, atoms, kind, layer in _linears(SHAPES[case["shape"]], case["layers"]):
        yield name, rows, cols, kind, layer, _parts(gen, rows, cols, 0, atoms, 8)


def _tokens(case, seed):
    """[batch][context + steps] token ids, uniform over the vocabulary."""
    n = case["context"] + case["steps"] if case["kind"] == "step" else case["tokens"]
    return np.random.default_rng(seed).integers(0, SHAPES[case["shape"]]["vocab"], (case.get("batch", 1), n)).astype(np.int32)


def _text(s):
    return struct.pack("<I", len(s)) + s.encode()


def _write_archive(path, case, seed):
    """A .sdr archive (version 2) of the decoder: every linear compressed, norm vectors stored raw."""
    hidden, index = SHAPES[case["shape"]]["hidden"], []
    with open(path, "wb") as f:
        f.write(b"CORTEXSR" + bytes(20))

        def put(name, payload, strategy, kind, dims, layer, words):
            n = payload.nbytes
            entry = _text(name) + _text("f32") + _text("LINEAR" if len(dims) == 2 else "")
            entry += struct.pack("<BBQQQ", kind, strategy, 4 * int(np.prod(dims)), n, f.tell()) + _text(name)
            entry += struct.pack("<IBB", layer, 1, len(dims)) + struct.pack("<%dI" % len(dims), *dims) + struct.pack("<fBBB", 0.0, 0, 0, 0)
            index.append(entry + words)
            f.write(memoryview(payload))

        norms = ["output_norm.weight"] + ["blk.%d.%s_norm.weight" % (i, n) for i in range(case["layers"]) for n in ("attn", "ffn")]
        for name in norms:
            put(name, np.ones(hidden, np.float32).view(np.uint8), 0, 14, (hidden,), 0, struct.pack("<BB", 0, 0))
        for name, rows, cols, kind, layer, parts in _decoder_parts(case, seed):
            put(name, _payload(parts, rows, cols, 0, 8), 5, kind, (rows, cols), layer,
                struct.pack("<BBII", 1, 2, 1, cols) + struct.pack("<BBII", 1, 2, 1, rows))
        at = f.tell()
        f.write(b"".join(index))
        f.seek(8)
        f.write(struct.pack("<IQQ", 2, len(index), at))


def _prepare_decoder(case, seed):
    spec, tokens = SHAPES[case["shape"]], _tokens(case, seed)
    handle, path = tempfile.mkstemp(suffix=".sdr")
    os.close(handle)
    try:
        _write_archive(path, case, seed)
        loader = cs.SDRModelLoader(path)
        dec = cs.Decoder(loader, n_layers=case["layers"], max_seq=tokens.shape[1] + 1, max_batch=tokens.shape[0], rms_eps=spec["eps"],
                         rope_theta=ROPE_THETA, **{k: spec[k] for k in ("hidden", "q_heads", "kv_heads", "head_dim", "inter", "vocab")})
    finally:
        os.unlink(path)
    if case["kind"] == "step":
        for s in range(tokens.shape[0]):
            dec.forward(tokens[s, :case["context"]], s, want_logits=False)
        given = [np.ascontiguousarray(tokens[:, case["context"] + i]) for i in range(case["steps"])]
        return dict(kind="step", dec=dec, given=given, context=case["context"])
    return dict(kind="prompt", dec=dec, tokens=np.ascontiguousarray(tokens[0]))


def _run_decoder(s):
    if s["kind"] == "prompt":
        s["dec"].seek(0, 0)
        return list(s["dec"].forward(s["tokens"], 0, True, True))
    for i in range(s["given"][0].size):
        s["dec"].seek(i, s["context"])
    return [s["dec"].step(t, want_logits=True)[1] for t in s["given"]]


def _exact_decoder(case, seed):
    spec, tokens = SHAPES[case["shape"]], torch.from_numpy(_tokens(case, seed).astype(np.int64)).cuda()
    batch, n = tokens.shape
    hd, qh, kh = spec["head_dim"], spec["q_heads"], spec["kv_heads"]

    def norm(x):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + spec["eps"])

    freq = torch.tensor(ROPE_THETA, dtype=torch.float64, device="cuda") ** (-torch.arange(0, hd, 2, device="cuda").double() / hd)
    angle = torch.arange(n, device="cuda").double()[:, None] * freq

    def rope(x):  # [tokens][heads][head_dim], adjacent pairs
        c, s = angle.cos()[:, None], angle.sin()[:, None]
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)

    def attend(q, k, v):
        q, k, v = rope(q.view(n, qh, hd)).transpose(0, 1), rope(k.view(n, kh, hd)).transpose(0, 1), v.view(n, kh, hd).transpose(0, 1)
        out = []
        for h in range(qh):
            g = h // (qh // kh)
            sc = (q[h] @ k[g].T) / math.sqrt(hd)
            sc.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), -math.inf)
            out.append(sc.softmax(-1) @ v[g])
        return torch.stack(out, 1).reshape(n, qh * hd)

    stream = _decoder_parts(case, seed)

    def weight():
        _, rows, cols, _, _, parts = next(stream)
        return _dense(parts, rows, cols, 0, 8)

    x = weight()[tokens]
    for _ in range(case["layers"]):
        y = norm(x)
        q, k, v = (y @ weight().T for _ in range(3))
        x = x + torch.stack([attend(q[b], k[b], v[b]) for b in range(batch)]) @ weight().T
        y = norm(x)
        g = torch.nn.functional.silu(y @ weight().T)
        x = x + (g * (y @ weight().T)) @ weight().T
    x, head = norm(x), weight()
    if case["kind"] == "prompt":
        return [x[0, -1] @ head.T, x[0]]
    return [x[:, case["context"] + i] @ head.T for i in range(case["steps"])]


# ---- the interface ----

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("product", "group", "list"):
        return _prepare_product(case, seed)
    if kind in ("step", "prompt"):
        return _prepare_decoder(case, seed)
    gen = _generator(seed)
    if kind == "encode":
        w = torch.randn(case["rows"], case["cols"], generator=gen, device="cuda") * WEIGHT_STD
        return dict(kind=kind, strategy=cs.HierarchicalSDRStrategy(), w=w.cpu().numpy(),
                    options=dict(tile_rows=1, tile_cols=case["cols"], n_atoms=case["atoms"], n_stages=STAGES, k=case["k"]))
    parts = _parts(gen, case["rows"], case["cols"], case["tile"], case["atoms"], case["k"])
    seg = cs.Segment.from_payload(_payload(parts, case["rows"], case["cols"], case["tile"], case["k"]))
    return dict(kind=kind, seg=seg, out=torch.empty(case["rows"], case["cols"], device="cuda"))


def run(state):
    kind = state["kind"]
    if kind in ("product", "group", "list"):
        return _run_product(state)
    if kind in ("step", "prompt"):
        return _run_decoder(state)
    if kind == "encode":
        return np.frombuffer(state["strategy"].compress(state["w"], **state["options"]), np.uint8)
    state["seg"].decompress_device(state["out"].data_ptr())
    return state["out"]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("product", "group", "list"):
        return _exact_product(case, seed)
    if kind in ("step", "prompt"):
        return _exact_decoder(case, seed)
    if kind == "encode":
        return None
    parts = _parts(_generator(seed), case["rows"], case["cols"], case["tile"], case["atoms"], case["k"])
    return _dense(parts, case["rows"], case["cols"], case["tile"], case["k"])


def work(case):
    kind = case["kind"]
    if kind in ("step", "prompt"):
        spec, n = SHAPES[case["shape"]], case["layers"]
        linears, qd, kd = _linears(spec, n), spec["q_heads"] * spec["head_dim"], spec["kv_heads"] * spec["head_dim"]
        weights = sum(_payload_bytes(r, c, 0, a, 8) for _, r, c, a, _, _ in linears[1:])
        macs = sum(a * c + r * STAGES * 8 / 2 for _, r, c, a, _, _ in linears[1:-1])
        _, r, c, a, _, _ = linears[-1]
        head = a * c + r * STAGES * 8 / 2
        if kind == "step":
            b, s, seen = case["batch"], case["steps"], case["context"] + (case["steps"] + 1) / 2
            return dict(bytes=s * (weights + n * b * seen * kd * 8 + b * spec["vocab"] * 4),
                        flops=2 * s * b * (macs + head) + s * b * n * seen * qd * 4)
        t = case["tokens"]
        return dict(bytes=weights + n * t * kd * 8 + t * spec["hidden"] * 4 + spec["vocab"] * 4,
                    flops=2 * (t * macs + head) + n * t * (t + 1) / 2 * qd * 4)
    rows, cols, k, atoms = case["rows"], case["cols"], case["k"], case["atoms"]
    slots = STAGES * k
    if kind == "encode":
        return dict(bytes=rows * cols * 4 + _payload_bytes(rows, cols, 0, atoms, k), flops=2.0 * rows * atoms * cols + 2.0 * atoms * atoms * cols + rows * slots * atoms)
    tile = case["tile"]
    if kind == "decompress":
        return dict(bytes=_payload_bytes(rows, cols, tile, atoms, k) + rows * cols * 4, flops=2.0 * rows * cols * slots)
    m, xb = case["batch"], 2 if case["dtype"] == "bf16" else 4
    n, n_x = case["members"], case["members"] if kind == "list" else 1
    if tile:  # all tile products once and a gather of rows, or the weight rebuilt and a dense product
        flops = min(2.0 * atoms * tile * cols * m + 1.0 * rows * (cols // tile) * slots * m, rows * cols * (slots + 2.0 * m))
    else:
        flops = 2.0 * atoms * cols * m + 1.0 * rows * slots * m
    return dict(bytes=n * (_payload_bytes(rows, cols, tile, atoms, k) + rows * m * 4) + n_x * cols * m * xb, flops=n * flops)


def tolerance(case):
    kind = case["kind"]
    if kind == "decompress":   # one multiplication and one addition per code, in code order: the same bits everywhere
        return "exact"
    if kind == "encode":       # where two projections tie within rounding another atom may be picked
        return {"rel": 0.0, "differ": 0.01}
    if kind in ("step", "prompt"):   # four times the 6e-5 that blocks of 16-bit splits are off from 64 bits
        return {"rel": 2.5e-4}
    return {"rel": 4e-5}             # four times the 1e-5 of a product over 16-bit splits of both operands

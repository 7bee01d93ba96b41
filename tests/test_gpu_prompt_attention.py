"""Attention of a prompt block by block (CSDR_PROMPT_ATTENTION_MIN) against the kernel that walks the
cache once per token: grouped heads, both head sizes, every cache type, prompts around the 64-row and
64-key blocks, with and without a context before them."""
import numpy as np
import pytest

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


def archive(path, head_dim, q_heads, kv_heads, raw=None):
    cfg = dict(n_layers=2, hidden=128, q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, inter=256, vocab=128)
    synth.decoder_archive(str(path), **cfg, n_atoms=128, k=4, raw=raw)
    return cfg


def hidden_states(path, cfg, monkeypatch, least, kv_dtype, passes, max_seq=300):
    monkeypatch.setenv("CSDR_PROMPT_ATTENTION_MIN", str(least))
    ctx = cs.Context(0)
    ld = cs.SDRModelLoader(str(path), ctx)
    dec = cs.Decoder(ld, **cfg, max_seq=max_seq, max_batch=2, kv_dtype=kv_dtype)
    out = [dec.forward(p, 1, want_logits=False, want_hidden=True)[1] for p in passes]
    dec.close()
    ld.close()
    ctx.close()
    return out


@pytest.mark.parametrize("kv_dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("head_dim,q_heads,kv_heads", [(64, 3, 3), (64, 14, 2), (128, 2, 2), (128, 4, 1)])
def test_blocks_equal_the_walk(tmp_path, monkeypatch, head_dim, q_heads, kv_heads, kv_dtype):
    cfg = archive(tmp_path / "m.sdr", head_dim, q_heads, kv_heads)
    rng = np.random.default_rng(head_dim)
    passes = [rng.integers(0, 128, n) for n in (64, 1, 17, 129, 65)]      # contexts of 0, 64, 65, 82, 211
    walk = hidden_states(tmp_path / "m.sdr", cfg, monkeypatch, 10 ** 6, kv_dtype, passes)
    blocks = hidden_states(tmp_path / "m.sdr", cfg, monkeypatch, 2, kv_dtype, passes)
    for a, b in zip(walk, blocks):
        # fp32 sums in another order, then a 16-bit split of the next projection's input (2^-17 of each
        # element); with a 16-bit cache a key or value may round the other way in the second layer
        tol = 3e-5 if kv_dtype == "f32" else 1e-3 if kv_dtype == "f16" else 8e-3
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)


def test_a_later_token_that_is_not_finite_reaches_no_earlier_one(tmp_path, monkeypatch):
    cfg = archive(tmp_path / "m.sdr", 64, 4, 2, raw={"token_embd.weight": "f32"})
    at = cs.SDRModelLoader(str(tmp_path / "m.sdr"), index_only=True).findSegmentHeader("token_embd.weight").data_offset
    with open(tmp_path / "m.sdr", "r+b") as f:
        f.seek(at + 7 * 128 * 4)
        f.write(np.full(128, np.nan, np.float32).tobytes())               # token 7
    tokens = np.full(100, 3)
    tokens[70] = 7
    (h,) = hidden_states(tmp_path / "m.sdr", cfg, monkeypatch, 2, "f32", [tokens])
    assert np.isfinite(h[:70]).all() and np.isnan(h[70:]).all()

"""Decode steps with the norms folded into the GEMVs give those of the separate kernels whatever the
dictionaries' sizes (the norm weights lie in shared memory behind slices of any number of atoms)."""
import numpy as np
import pytest

import cortexsdr_b200 as cs
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms", [30, 33, 64])
@pytest.mark.parametrize("batch", [1, 2, 3])
def test_folded_steps(tmp_path, monkeypatch, atoms, batch):
    cfg = dict(n_layers=2, hidden=128, q_heads=4, kv_heads=2, head_dim=32, inter=256, vocab=128)
    synth.decoder_archive(str(tmp_path / "m.sdr"), **cfg, n_atoms=atoms, k=4)
    tokens = np.random.default_rng(atoms).integers(0, 128, (4, batch)).astype(np.int32)
    out = []
    for fold in ("1", "0"):
        monkeypatch.setenv("CSDR_DECODER_FOLD", fold)
        ctx = cs.Context(0)
        ld = cs.SDRModelLoader(str(tmp_path / "m.sdr"), ctx)
        dec = cs.Decoder(ld, **cfg, max_seq=16, max_batch=batch)
        out.append([dec.step(t, want_logits=True)[1] for t in tokens])
        dec.close()
        ld.close()
        ctx.close()
    for a, b in zip(*out):
        # fp32 throughout, the factor 1 / rms on the other side of the sums
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)

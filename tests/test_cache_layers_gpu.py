"""The radiance cache's encoding and layers on the GPU where their arithmetic changes form: arguments of
any size in the encoding, and tile, group and CTA edges of the tcgen05 kernel."""
import numpy as np
import pytest

from oracle import nrc_oracle as nrc
from trenchanttracer_gb300 import Cache

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LO, HI = (-2.0, 0.0, -1.0), (2.0, 4.0, 3.0)  # extents of 4: the normalised position is exact in FP32


def _records(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    rec = np.zeros((n, 16), np.float32)
    rec[:, 0:3] = np.array(LO) + 4.0 * scale * rng.random((n, 3))
    for c in (3, 6):
        d = rng.standard_normal((n, 3))
        rec[:, c:c + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec[:, 9:13] = rng.random((n, 4))
    rec[:, 13] = rng.integers(0, 6, n) / 8.0
    return rec


@pytest.mark.parametrize("scale", [1.0, -1.0, 1e3, -1e4, 1e6, -1e8])
def test_encoding_of_positions_in_and_far_outside_the_box(scale):
    """sin and cos of pi 2^k p for FP32 p, reduced in FP64 (exact) before NumPy's sin and cos. The hardware
    approximations are within 1e-6 on the reduced argument, and BF16 rounds within 2^-9 relatively."""
    rec = _records(512, 3, scale)
    rec[:8, 0] = LO[0] + np.array([0, 1, 2, 4, 6, 8, 4096, -4096], np.float32)  # whole and half turns
    cache = Cache(LO, HI, batch=1024)
    got = cache.encode(torch.from_numpy(rec).cuda()).float().cpu().numpy().astype(np.float64)
    p = ((rec[:, :3] - np.float32(LO)) * np.float32(0.25)).astype(np.float64)
    for k in range(12):
        turn = np.pi * np.fmod(p * 2.0 ** k, 2.0)
        for o, ref in ((0, np.sin(turn)), (1, np.cos(turn))):
            err = np.abs(got[:, [24 * i + 2 * k + o for i in range(3)]] - ref)
            assert np.all(err <= 2.0 ** -8 * np.abs(ref) + 2e-6), (k, o, err.max())


@pytest.mark.parametrize("n", [1, 127, 128, 129, 5 * 128 + 1, 152 * 5 * 128 + 130])
def test_tcgen05_inference_matches_mma_sync(n):
    """Radiance of both kernels from the same BF16 weights and inputs; sums in another order move a BF16
    activation by a step (2^-8) now and then, as between any two of the cache's kernels."""
    w = nrc.init_weights(5)
    rec = torch.from_numpy(_records(n, 4)).cuda()
    out = []
    for kind in (0, 1):
        c = Cache(LO, HI, batch=4096, mma_kind=kind)
        c.set_weights(w)
        out.append(c.infer(rec).cpu().numpy())
        c.check()
    rel = np.abs(out[0] - out[1]) / np.abs(out[1])
    assert out[0].shape == (n, 3) and np.median(rel) < 1e-3 and np.quantile(rel, 0.999) < 5e-2

"""The radiance cache's tcgen05 kernels where a warpgroup goes on to its next tile of 128 rows and where training changes
its launch shape: sizes from the SM count and the kernels' groups per CTA, against the mma.sync kernels with the tolerances
of the cache's other comparisons of the two."""
import numpy as np
import pytest

from oracle import nrc_oracle as nrc
from tests.test_cache_gpu import HI, LO, _records, _target
from trenchanttracer_gb300 import Cache

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

INFER_GROUPS, TRAIN_GROUPS, TILE = 6, 5, 128  # warpgroups per CTA: inference, training of large batches


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tiles,rows", [(1, -1), (1, 0), (1, 1), (2, 130), (3, -1)])
def test_inference_over_several_tiles_a_group(tiles, rows):
    """tiles rounds of every group of every CTA (1: of one CTA), and some rows more or fewer."""
    n = TILE * INFER_GROUPS * (tiles * sms() if tiles > 1 else 1) + rows
    rec = torch.from_numpy(_records(n, 14)).cuda()
    w = nrc.init_weights(21)
    out = []
    for kind in (0, 1):
        c = Cache(LO, HI, batch=4096, mma_kind=kind)
        c.set_weights(w)
        out.append(c.infer(rec).cpu().numpy())
        c.check()
    rel = np.abs(out[0] - out[1]) / np.abs(out[1])
    assert np.median(rel) < 1e-3 and np.quantile(rel, 0.999) < 5e-2
    # the last rows of the last tiles as well as the first
    assert np.median(rel[-257:]) < 1e-3 and np.median(rel[:257]) < 1e-3


# two CTAs of one group to an SM, two threads a row: their second and third tiles; from TRAIN_GROUPS tiles per SM
# on CTAs of five groups: the last size before, the first, and their second tiles
@pytest.mark.parametrize("per_sm,rows", [(2, 129), (4, 1), (TRAIN_GROUPS, -TILE), (TRAIN_GROUPS, 0), (2 * TRAIN_GROUPS, 77)])
def test_training_over_several_tiles_a_group(per_sm, rows):
    n = TILE * per_sm * sms() + rows
    w = nrc.init_weights(31)
    rec = _records(n, 18)
    rec_t, tgt_t = torch.from_numpy(rec).cuda(), torch.from_numpy(_target(rec)).cuda()
    grads, losses = [], []
    for kind in (0, 1):
        c = Cache(LO, HI, batch=n, mma_kind=kind)
        c.set_weights(w)
        g, loss = c.gradient(rec_t, tgt_t)
        c.check()
        grads.append(g)
        losses.append(loss)
    assert abs(losses[0] - losses[1]) <= 1e-3 * losses[1]
    off = nrc.offsets()
    for l in range(nrc.LAYERS):
        a, b = (g[off[l]:off[l + 1]] for g in grads)
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 2e-2, l
    assert not grads[0][off[5] + 3 * 64:].any()

"""Float ground truth where the BF16 halves of the rows are as wrong as they can be: the
nearest point's score comes out low by all that the halves leave out, those of its rivals
high, and the true distances are close.  The screen's bound must keep the nearest point."""
import numpy as np
import pytest

from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _halves(metric, d, rivals, scale):
    """x = 1 + 2^-8 - 2^-17 -+ 2^-23: its upper half is 1 and leaves 2^-8, of which the
    lower one leaves 2^-17; the rivals' upper half is 1 + 2^-7, and both remainders are
    negative.  A second coordinate makes the first point the nearer one by a little."""
    e = 2.0 ** -23
    up = 1 + 2.0 ** -8 - 2.0 ** -17 - e
    down = 1 + 2.0 ** -8 + 2.0 ** -17 + e
    f = 1.0 if metric == "mips" else 2.0  # L2: a query beyond the points
    q = np.zeros(d)
    q[0], q[1] = f * up, f * 2.0 ** -4
    step = 2.0 ** -12 * (1 + 2.0 ** -5) if metric == "mips" else 2.0 ** -13 * (1 + 2.0 ** -5)
    near = np.zeros(d)
    near[0], near[1] = up, step
    far = np.zeros(d)
    far[0] = down
    # farther points fill tiles; the near ones lie in different ones
    rng = np.random.default_rng(d)
    n = 700
    base = np.zeros((n, d))
    base[:, 0] = -rng.random(n)
    at = [390] + list(range(5, 5 + rivals))
    base[at[0]] = near
    base[at[1:]] = far
    return (np.float32(scale) * base.astype(np.float32), np.float32(scale) * q[None].astype(np.float32),
            at[0])


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 2.0 ** 30])
@pytest.mark.parametrize("rivals", [1, 12, 40])
@pytest.mark.parametrize("metric,d", [("mips", 2), ("mips", 3), ("l2", 2), ("l2", 3)])
def test_worst_halves(oracle_mod, metric, d, rivals, scale):
    base, q, near = _halves(metric, d, rivals, scale)
    gi = GpuIndex(np.float32, metric, base.shape[0], d, 8)
    gi.upload_points(base)
    for k in (1, 5, 32):
        oi, od = oracle_mod.groundtruth(base, q, k, metric=metric)
        assert oi[0, 0] == near
        ids, ds = gi.groundtruth(q, k)
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(ds, od)
    gi.close()

"""The packed quantiser of the compressor against the oracle where its roundings meet: at halves and whole numbers of steps, one
and two floats to either side, both signs, over all magnitudes that take the float form and beyond."""
import numpy as np
import pytest
import torch

from tirocinio_triennale_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eb", [0.5, 1e-3, 1e-4, 3e-7, 2.0 ** 60])
def test_ties_whole_numbers_and_their_neighbours(eb):
    rng = np.random.default_rng(1)
    m = np.concatenate([np.arange(0, 4096), rng.integers(0, 2 ** rng.integers(1, 25, 60_000))])
    t = np.concatenate([m, m + 0.5]).astype(np.float64)
    x = (t * 2 * np.float64(np.float32(eb))).astype(np.float32)
    near = [x, -x]
    for toward in (np.float32(-np.inf), np.float32(np.inf)):
        y = x
        for _ in range(2):
            y = np.nextafter(y, toward)
            near += [y, -y]
    x = np.concatenate(near)
    x = x[np.lexsort((x, np.abs(x)))]  # neighbours of like magnitude: blocks stay in the float form
    for values in (x, x[rng.permutation(x.size)], np.concatenate([x[:100], np.float32([0.0, -0.0, 1e-45, -1e-45]), x[-999:]])):
        want = ops.cpu_compress(values, eb)
        c = ops.Codec(values.size)
        out, size = c.compress(torch.from_numpy(values).cuda(), eb)
        assert int(size) == want.size
        np.testing.assert_array_equal(out[:want.size].cpu().numpy(), want)
        assert c.status() == 0

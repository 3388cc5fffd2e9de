"""The row-ring convolution (x-rows of 128 nodes) at the shortest and odd counts of planes and row
groups, with one chunk of input channels and several, with 16 and more channels out (256 nodes: the
second level's rows hold 128), and the features of sources outside the grid: predictions against the
network in FP64, as close as the oracle's BF16 emulation of it is (twice its distance: the rounding
noise at this depth; a product of a wrong row or tap is a hundred times that)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from eikonalxx_gb300 import warmstart as ws  # noqa: E402
from oracle import warmnet_oracle as wo  # noqa: E402
from test_gpu_warmnet import _device, _host_samples, _params  # noqa: E402


def _grid(nx, ny, nz):
    return (nx, ny, nz, 50.0, 50.0, 50.0, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("shape,count", [((128, 8, 8), 1), ((128, 24, 40), 3), ((256, 16, 24), 2)])
@pytest.mark.parametrize("outside", [False, True])
def test_prediction_matches_the_oracle_at_edges(shape, count, outside):
    grid = _grid(*shape)
    host = _host_samples(21, count, grid)
    if outside:
        host = [(v, t, (s[0], -30.0, s[2])) for v, t, s in host]
    p = _params(9)
    with ws.WarmNet(grid, batch=count, seed=0) as net:
        net.set_params(p)
        t, _ = net.predict(_device(host), inflate=1.0)
    exact, emulated = (wo.predict(p, host, grid, emulate=e) for e in (False, True))
    noise = np.linalg.norm(emulated - exact)
    assert np.linalg.norm(t - exact) <= 2 * noise
    assert np.linalg.norm(t - emulated) <= 2 * noise

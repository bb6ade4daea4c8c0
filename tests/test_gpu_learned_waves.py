"""The learned time-block kernel's two sizes (fewer or more resident CTAs, chosen
by the number of waves of the grid) give the same bits: a few particles alone,
and the same particles repeated to a grid that the larger size takes in one
wave and the smaller in two, and one beyond both."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
import perf.cases as K  # noqa: E402
from test_smallstep_host import DT, MU, states  # noqa: E402

BASE, STEPS = 640, 5


@pytest.fixture(scope="module")
def network():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()
    tr = K._trainer(20_000, 5)
    tr.train(200, batch=2048, lr=1e-2, seed=3)
    return tr


@pytest.mark.parametrize("ctas_per_sm", [15, 17])
@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
def test_a_particles_path_does_not_depend_on_the_grid(network, ctas_per_sm, kick):
    from gpu_util import DevHandoff, DevParticles, DevPlanetBlock, timeblock
    rng = np.random.default_rng(41)
    # all tiers of the drift, the network's (tau^2 >= 0.01) the most
    rv = states(np.exp(rng.uniform(np.log(1e-4), np.log(0.3), BASE)), rng.uniform(0, 0.5, BASE), 42)
    out = []
    for n in (BASE, 64 * ctas_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 1):
        x = np.tile(rv, ((n + BASE - 1) // BASE, 1))[:n]
        p = DevParticles(x[:, :3], x[:, 3:], np.zeros((n, 3)), np.zeros(n), np.arange(n))
        b = DevPlanetBlock(np.zeros((STEPS, 3)), np.full((STEPS, 1, 3), 40.0), [MU, 1e-8], [0, 1], [0.01, 0.01])
        timeblock(p, b, DT, 1e6, starter=G.STARTER_LEARNED, handoff=DevHandoff(n), mlp=network.device_weights(), kick=kick)
        h = p.host()
        out.append(np.concatenate([h["r"], h["v"]], 1))
    assert np.array_equal(out[1], np.tile(out[0], (len(out[1]) // BASE + 1, 1))[:len(out[1])])

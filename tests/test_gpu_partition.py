"""The three-way partition at the edges of its tiles (256 particles) and ranges
(at most 456, of whole tiles): sizes around both, and sets of one category."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 513, 456 * 256 - 1, 456 * 256, 456 * 256 + 1, 912 * 256 + 300])
@pytest.mark.parametrize("flags_of", ["mixed", "alive", "encounter", "dead"])
def test_partition_edges(n, flags_of):
    from gpu_util import DevParticles
    rng = np.random.default_rng(n)
    kinds = {"mixed": [0, 0, 0, 0x0401, 0x0080, 0x0002, 0x0001], "alive": [0], "encounter": [0x0301],
             "dead": [0x0080, 0x0002]}[flags_of]
    flags = rng.choice(kinds, n).astype(np.uint16)
    ids = rng.permutation(n).astype(np.uint32)
    r, v, a = (rng.normal(size=(n, 3)) for _ in range(3))
    src = DevParticles(r, v, a, flags, ids)
    src.dti.copy_(torch.arange(n, dtype=torch.int32))
    dst = DevParticles(r * 0, v * 0, a * 0, flags * 0, ids * 0)
    scratch = torch.zeros(G.partition_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    counts = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    G.partition(src.view, dst.view, n, scratch.data_ptr(), counts.data_ptr(), counts.data_ptr() + 4)
    out = dst.host()
    cat = np.where(flags == 0, 0, np.where((flags & 0xFE) == 0, 1, 2))
    order = np.argsort(cat, kind="stable")
    for k, x in (("r", r), ("v", v), ("a", a), ("flags", flags), ("id", ids), ("dti", np.arange(n, dtype=np.uint32))):
        assert np.array_equal(out[k], x[order]), k
    assert counts.cpu().tolist() == [(cat == 0).sum(), (cat == 1).sum()]

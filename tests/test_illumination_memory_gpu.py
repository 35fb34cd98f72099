"""Memory that source illumination takes for its sums per shot."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("batch,shots", [(1, 1), (1, 3), (2, 2), (4, 4), (4, 6), (6, 6)])
@pytest.mark.parametrize("after_gradient", [False, True])
def test_illumination_keeps_what_its_sums_need(batch, shots, after_gradient):
    """On the handle stay the three images (12.3 MB a volume here) and three sums
    for each shot of a batch after the first, up to four shots; a handle that has
    run a gradient has room for both."""
    from efwi.engine import Grid, Propagator, Shot
    g = Grid(96, 160, 200, 8, 8, 10.0, 10.0, 10.0, 8e-4, 25.0)
    one = torch.ones(g.shape)
    r = np.arange(20, 60, dtype=np.int32)
    every = [Shot(src=(40, 60 + k, 90), z_rec=0 * r + 12, x_rec=r, y_rec=r) for k in range(shots)]
    stf = np.random.default_rng(0).standard_normal((shots, g.nt)).astype(np.float32)
    P = Propagator(g, max_batch=batch)
    P.set_survey(every, stf)
    P.set_model(1.2e6 * one, 1e6 * one, 1.6 * one)
    ids = list(range(shots))
    obs = P.forward(ids)  # the state of a batch
    if after_gradient:
        P.gradient([0], obs[:sum(P.trace_sizes([0]))] + 1e-3)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    first = [t.cpu() for t in P.illumination(ids)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    sums = 3 * (batch - 1) if batch <= 4 else 0
    volumes = 0 if after_gradient else 3 + sums
    # (without the adjoint fields at all after a batch beyond them)
    assert free - torch.cuda.mem_get_info()[0] <= volumes * 4 * g.nz * g.nx * g.ny + 8 * MB
    for u, v in zip(first, P.illumination(ids)):
        assert float(u.max()) > 0 and torch.equal(u, v.cpu())
    P.close()

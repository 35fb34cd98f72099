"""The checkpoint budget of the exact gradient bounds the memory of the slots,
on grids whose rows are padded (ny 84 -> 96) as on others."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _engine(nt, lanes=1, ny=84):
    from efwi.engine import Grid, Propagator, Shot
    g = Grid(56, 57, ny, 8, nt, 10.0, 10.0, 10.0, 8e-4, 25.0)
    rng = np.random.default_rng(3)
    rho = (1.5 + rng.random(g.shape)).astype(np.float32)
    mu = (1e6 * (1.0 + rng.random(g.shape))).astype(np.float32)
    r = np.arange(10, 40, dtype=np.int32)
    shots = [Shot(src=(20, 28, 40), z_rec=0 * r + 12, x_rec=r, y_rec=r),
             Shot(src=(24, 20, 30), z_rec=0 * r + 12, x_rec=r, y_rec=r)]
    P = Propagator(g)
    P.set_lanes(lanes)
    P.set_survey(shots, rng.standard_normal((2, nt)).astype(np.float32))
    P.set_model(torch.from_numpy(1.2 * mu), torch.from_numpy(mu), torch.from_numpy(rho))
    n = sum(P.trace_sizes([0, 1]))
    w = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    return P, w


def _unpadded_bytes(g):
    pml = 12 * g.npml * (g.nx * g.ny + g.nz * g.ny + g.nz * g.nx)
    return 4 * (9 * g.nz * g.nx * ((g.ny + 3) // 4 * 4) + pml)


@pytest.mark.parametrize("lanes", [1, 2])
@pytest.mark.parametrize("ny", [84, 90, 66])
def test_slots_take_no_more_than_the_budget(lanes, ny):
    nt, n = 60, 16
    P, w = _engine(nt, lanes, ny)
    state = P.state_bytes()
    assert state == _unpadded_bytes(P.grid)
    # everything but the slots is allocated by a call with room for two states a lane
    P.set_checkpoint_budget(2 * lanes * state)
    few = P.gradient([0, 1], w, mode="exact")[1:]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0] + 2 * lanes * state
    P.set_checkpoint_budget(n * lanes * state)
    many = P.gradient([0, 1], w, mode="exact")[1:]
    torch.cuda.synchronize()
    assert P.checkpoint_stats()["slots"] == n
    # allocations come in granules of 2 MB, two buffers a lane at most; 16 states
    # with padded rows would be 22 MB over
    assert free - torch.cuda.mem_get_info()[0] <= n * lanes * state + 8 * MB
    for u, v in zip(few, many):
        assert torch.equal(u, v)


@pytest.mark.parametrize("ny", [84, 90])
@pytest.mark.parametrize("variant", [0, 1])
def test_schedules_of_padded_grids_give_the_same_images(ny, variant):
    """Rows of 84 and 92 cells in the slots, of 96 in the work buffers: every
    state kept, one, and a few (steps from slot to slot, from and to the work
    buffers)."""
    nt = 31
    P, w = _engine(nt, 1, ny)
    P.set_variant(variant)
    ref = None
    for n in (nt, 1, 2, 5, 12):
        P.set_checkpoint_budget(n * P.state_bytes())
        out = list(P.gradient([0, 1], w, mode="exact")[1:]) + list(P.adjoint([0, 1], w))
        ref = ref or out
        for u, v in zip(ref, out):
            assert float(u.abs().max()) > 0
            assert torch.equal(u, v)

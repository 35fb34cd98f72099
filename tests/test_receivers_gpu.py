"""Receivers on the cells that a time step does not update (the outer two of
each side): the reference gradient injects their residual (minus the observed
data; their traces are zero) into the adjoint velocities there, which the
adjoint stresses beside them read.  Both kernel families give the same bits,
also for a window whose edge cuts through the receivers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _problem(nz, nx, ny, npml, nt=40):
    from efwi.engine import Grid, Shot
    g = Grid(nz, nx, ny, npml, nt, 10.0, 11.0, 9.0, 8e-4, 25.0)
    rng = np.random.default_rng(nz + ny)
    rho = (1.5 + rng.random((nz, nx, ny))).astype(np.float32)
    mu = (1e6 * (1.0 + rng.random((nz, nx, ny)))).astype(np.float32)
    model = [torch.from_numpy(a) for a in ((1.2 * mu).astype(np.float32), mu, rho)]
    shots = []
    for k, edge in enumerate((0, 1, 2)):  # a shot's receivers: all inside, on one face, anywhere
        z, x, y = (rng.integers(2, n - 2, 30 + 10 * k).astype(np.int32) for n in (nz, nx, ny))
        if edge == 1:
            y[:12] = ny - 2
        if edge == 2:
            z, x, y = (rng.integers(0, n, 50).astype(np.int32) for n in (nz, nx, ny))
        shots.append(Shot(src=(nz // 2, nx // 2, ny // 2), z_rec=z, x_rec=x, y_rec=y))
    return g, shots, rng.standard_normal((3, nt)).astype(np.float32), model


def _engine(g, shots, stf, model, variant, graphs, lanes):
    from efwi.engine import Propagator
    P = Propagator(g)
    P.set_variant(variant)
    P.set_graphs(graphs)
    P.set_lanes(lanes)
    P.set_survey(shots, stf)
    P.set_model(*model)
    return P


@pytest.mark.parametrize("size", [(14, 13, 12, 4), (17, 18, 35, 6), (61, 70, 66, 7)])
@pytest.mark.parametrize("graphs,lanes", [(True, 1), (False, 1), (True, 2)])
def test_reference_gradient_with_outer_receivers(size, graphs, lanes):
    case = _problem(*size)
    out = []
    for variant in (0, 1):
        P = _engine(*case, variant, graphs, lanes)
        n = sum(P.trace_sizes([0, 1, 2]))
        obs = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
        J, *grads = P.gradient([0, 1, 2], obs)
        out.append([torch.tensor(J)] + grads)
        # each shot alone on the same handle: receiver counts of every kind in turn
        off = 0
        for k in (0, 1, 2, 1):
            size_k = sum(P.trace_sizes([k]))
            off = sum(P.trace_sizes(list(range(k))))
            out[-1] += P.gradient([k], obs[off:off + size_k])[1:]
    for u, v in zip(*out):
        assert float(u.abs().max()) > 0
        assert torch.equal(u, v)


def test_window_gradient_with_receivers_on_its_edge():
    g, shots, stf, model = _problem(24, 40, 48, 4)
    wins = [(4, 5, 30, 36), (6, 8, 28, 32), (2, 4, 33, 40)]
    x0, y0, nx, ny = wins[0]
    shots[0].x_rec[:6], shots[0].y_rec[:6] = x0 + 1, np.arange(10, 16)
    shots[0].y_rec[6:9] = y0 + ny - 1
    out = []
    for variant in (0, 1):
        P = _engine(g, shots, stf, model, variant, True, 1)
        n = sum(P.trace_sizes([0, 1, 2]))
        obs = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(8))
        J, *grads = P.gradient_windows([0, 1, 2], wins, obs)
        out.append([torch.tensor(J)] + grads)
    for u, v in zip(*out):
        assert float(u.abs().max()) > 0
        assert torch.equal(u, v)


def test_receiver_cells_of_shots_in_turn_beyond_the_launch_limits():
    """More planes than one launch of the vector kernels takes: the one-cell
    kernels run, and the captured time loop's separate receiver launch covers
    the cells of the shot at hand (3, then 30, for as many receivers)."""
    from efwi.engine import Grid, Propagator, Shot
    nz, n, nt = 4 * 65535 + 20, 30, 24
    g = Grid(nz, 5, 5, 2, nt, 10.0, 10.0, 10.0, 8e-4, 25.0)
    model = [torch.full((nz, 5, 5), v) for v in (1.2e6, 1e6, 1.6)]
    two = np.full(n, 2, np.int32)
    shots = [Shot(src=(nz // 2, 2, 2), z_rec=(nz // 2 - 15 + r % cells).astype(np.int32), x_rec=two,
                  y_rec=two) for cells, r in ((3, np.arange(n)), (n, np.arange(n)))]
    stf = np.random.default_rng(0).standard_normal((2, nt)).astype(np.float32)
    out = []
    for graphs in (False, True):
        P = Propagator(g)
        P.set_graphs(graphs)
        P.set_survey(shots, stf)
        P.set_model(*model)
        out.append([P.forward([k]).view(3, n, nt) for k in (0, 1, 0)])
        P.close()
    for u, v in zip(*out):
        assert torch.equal(u, v)
    assert bool((out[1][1][2].abs().amax(1) > 0).all())

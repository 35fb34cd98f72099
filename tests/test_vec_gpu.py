"""Vector kernels (variant 1, four cells per thread) against the one-cell
L1 kernels (variant 0): the same bits, at the edges of their vectors, tiles
and slabs.  ny runs over every remainder by the vector length; C-PML widths
and ny that are not multiples of it take the single-cell memory variables,
the others the vector ones; nx and nz run over the remainders of the 4 x 4
row and plane tile; the smallest grid has one updated cell.  On all but the last four grids the
forward kernels split their outputs over warps; the last two have rows of
whole lines."""
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
    for k in range(2):
        # receivers over all updated cells, C-PML and shared cells among them
        z, x, y = (rng.integers(2, n - 2, 40).astype(np.int32) for n in (nz, nx, ny))
        z[:5], x[:5], y[:5] = nz // 2, nx // 2, ny // 2
        shots.append(Shot(src=(2 + k * (nz - 5), nx // 2, 2 + (1 - k) * (ny - 5)), z_rec=z, x_rec=x,
                          y_rec=y))
    stf = rng.standard_normal((2, nt)).astype(np.float32)
    return g, shots, stf, model


SIZES = [(5, 5, 5, 2), (14, 13, 12, 4), (15, 14, 33, 4), (16, 17, 34, 5), (17, 18, 35, 6),
         (18, 19, 36, 8), (23, 22, 40, 4), (22, 23, 64, 8), (13, 24, 69, 6),
         (61, 70, 66, 7), (62, 71, 68, 8), (56, 57, 90, 5), (46, 61, 124, 8)]


def _run(g, shots, stf, model, obs, variant, graphs):
    from efwi.engine import Propagator
    P = Propagator(g)
    P.set_variant(variant)
    P.set_graphs(graphs)
    P.set_survey(shots, stf)
    P.set_model(*model)
    ids = list(range(len(shots)))
    tr = P.forward(ids)
    out = [tr] + list(P.gradient(ids, obs if obs is not None else 0.5 * tr + 1e-4)[1:])
    return out, list(P.illumination(ids))


@pytest.mark.parametrize("nz,nx,ny,npml", SIZES)
@pytest.mark.parametrize("graphs", [True, False])
def test_vector_kernels_match_single_cell_kernels(nz, nx, ny, npml, graphs):
    g, shots, stf, model = _problem(nz, nx, ny, npml)
    a, ia = _run(g, shots, stf, model, None, 0, graphs)
    b, ib = _run(g, shots, stf, model, None, 1, graphs)
    assert float(a[0].abs().max()) > 0
    for u, v in zip(a, b):
        assert torch.equal(u, v)
    # Sums of squares, over steps and then shots in one family and over shots
    # and then steps in the other: 80 additions of one sign and about 10
    # roundings a term, 90 * 2^-24 = 5e-6 at most, as much again for the terms
    # themselves (fused differently).
    for u, v in zip(ia, ib):
        assert float(u.max()) > 0
        assert float(torch.linalg.vector_norm(u - v)) <= 1e-5 * float(torch.linalg.vector_norm(u))


def test_illumination_in_batches_of_any_size():
    """Five shots in one batch (sums beyond the adjoint fields' memory), in
    batches of two and of one: sums of 5 * 40 squares, 2e-5."""
    from efwi.engine import Propagator
    g, shots, stf, model = _problem(22, 23, 36, 4)
    shots = [shots[k % 2] for k in range(5)]
    stf = np.concatenate([stf, 2 * stf, 3 * stf])[:5]
    out = []
    for batch in (5, 2, 1):
        P = Propagator(g, max_batch=batch)
        P.set_survey(shots, stf)
        P.set_model(*model)
        out.append(P.illumination(list(range(5))))
        grad = P.gradient([0], P.forward([0]) + 1e-4)[1:]
        assert all(float(t.abs().max()) > 0 for t in grad)
    for other in out[1:]:
        for u, v in zip(out[0], other):
            assert float(u.max()) > 0
            assert float(torch.linalg.vector_norm(u - v)) <= 2e-5 * float(torch.linalg.vector_norm(u))


@pytest.mark.parametrize("nz,nx,ny,npml", SIZES)
def test_exact_vector_kernels_match_single_cell_kernels(nz, nx, ny, npml):
    """The exact adjoint's sums have the same terms in both families but may
    be fused differently: about 20 roundings of 2^-24 a step, adding up at
    random over 40 steps to 2e-6; held to 5e-6 (rel-L2).  The first ten
    receivers lie anywhere, outside the updated cells too."""
    from efwi.engine import Propagator
    g, shots, stf, model = _problem(nz, nx, ny, npml)
    rng = np.random.default_rng(1)
    for s in shots:
        for a, n in ((s.z_rec, nz), (s.x_rec, nx), (s.y_rec, ny)):
            a[:10] = rng.integers(0, n, 10)
    out = []
    for variant in (0, 1):
        P = Propagator(g)
        P.set_variant(variant)
        P.set_survey(shots, stf)
        P.set_model(*model)
        n = sum(P.trace_sizes([0, 1]))
        gen = torch.Generator(device="cuda").manual_seed(5)
        w = torch.randn(n, device="cuda", generator=gen)
        P.set_checkpoint_budget(7 * P.state_bytes())
        out.append(list(P.adjoint([0, 1], w)) + list(P.gradient([0, 1], w, mode="exact")[1:]))
    for u, v in zip(*out):
        assert float(u.abs().max()) > 0
        assert float(torch.linalg.vector_norm(u - v)) <= 5e-6 * float(torch.linalg.vector_norm(u))

"""Kernel choices against one another where other tests do not reach them: the
prefetching of rows on grids whose working set is beyond L2 (20 volumes of more
than 64 MB in all), and the one-cell kernels' z planes per CTA."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _engine(size, npml, nt, variant, tile_bx=4, zchunk=8, **tuning):
    from efwi.engine import Grid, Propagator, Shot
    g = Grid(*size, npml, nt, 10.0, 11.0, 9.0, 8e-4, 25.0)
    rng = np.random.default_rng(sum(size))
    rho = (1.5 + rng.random(g.shape)).astype(np.float32)
    mu = (1e6 * (1.0 + rng.random(g.shape))).astype(np.float32)
    nz, nx, ny = size
    shots = []
    for k in range(2):  # near a corner and in the middle
        src = (4, 5, 6) if k else (nz // 2, nx // 2, ny // 2)
        z, x, y = (np.clip(c + rng.integers(-6, 7, 40), 2, n - 3).astype(np.int32)
                   for c, n in zip(src, size))
        shots.append(Shot(src=src, z_rec=z, x_rec=x, y_rec=y))
    P = Propagator(g, tile_bx=tile_bx, zchunk=zchunk)
    P.set_variant(variant)
    P.set_tuning(**tuning)
    P.set_survey(shots, rng.standard_normal((2, nt)).astype(np.float32))
    P.set_model(*[torch.from_numpy(a) for a in ((1.2 * mu).astype(np.float32), mu, rho)])
    return P


def _outputs(P):
    tr = P.forward([0, 1])
    return [tr] + list(P.gradient([0, 1], 0.5 * tr + 1e-4)[1:]), \
        list(P.gradient([0, 1], 0.5 * tr + 1e-4, mode="exact")[1:])


@pytest.mark.parametrize("size,npml", [((60, 100, 144), 8), ((61, 101, 141), 7)])
def test_vector_kernels_with_prefetching(size, npml):
    """Memory variables as vectors and as single cells.  Traces and reference
    images to the bit; exact images to 5e-6 (rel-L2), as on the small grids:
    about 20 roundings of 2^-24 a step in sums fused differently."""
    assert 20 * 4 * size[0] * size[1] * size[2] > 64 << 20
    (a, ea), (b, eb) = (_outputs(_engine(size, npml, 14, v)) for v in (0, 1))
    for u, v in zip(a, b):
        assert float(u.abs().max()) > 0
        assert torch.equal(u, v)
    for u, v in zip(ea, eb):
        assert float(u.abs().max()) > 0
        assert float(torch.linalg.vector_norm(u - v)) <= 5e-6 * float(torch.linalg.vector_norm(u))


@pytest.mark.parametrize("tile_bx", [4, 8])
@pytest.mark.parametrize("fwd,rev", [(1, 1), (3, 2), (5, 7), (64, 64)])
def test_planes_per_cta_of_the_one_cell_kernels(tile_bx, fwd, rev):
    size, npml = (23, 22, 39), 5
    ref = _outputs(_engine(size, npml, 40, 0))
    out = _outputs(_engine(size, npml, 40, 0, tile_bx, fwd, zchunk_fwd=fwd, zchunk_rev=rev))
    for a, b in zip(ref[0] + ref[1], out[0] + out[1]):
        assert float(a.abs().max()) > 0
        assert torch.equal(a, b)

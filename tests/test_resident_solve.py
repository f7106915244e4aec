"""The resident solve (csrc/cg_res.cuh) at the sizes where its tiling changes: one
tile and its remainders, the largest single cluster and one tile more, the last
size of each cluster form, the step to taller tiles, and the first shape that
falls back to the general kernel.

The systems are I + Laplacian with random face couplings and a tenth of the rows
decoupled.  The solve stops on its recursive residual, ||r|| < 1e-12 ||b||; the
true residual may exceed it by the recursion's rounding, at most about
iterations * 2^-53 * ||A|| ||x|| <= 60 * 1.1e-16 * 9 ||b|| = 6e-14 ||b|| here (the
smallest eigenvalue of A is 1), so 1.2e-12 ||b|| bounds it with room.
"""
import numpy as np
import pytest

from frehdc_b200 import deck as D
from frehdc_b200 import native
from tests.helpers import max_rel

pytestmark = pytest.mark.gpu

TILE = 16  # rows of the smallest tile (64 columns)


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if native.device_count() < 1:
        pytest.fail("no CUDA device visible: the GPU tests need a B200")


def _system(nx, ny):
    rng = np.random.default_rng([nx, ny])
    Gx, Gy = rng.uniform(0, 1, (ny, nx)), rng.uniform(0, 1, (ny, nx))
    Gx[:, -1] = 0
    Gy[-1] = 0
    Ct = 1 + Gx + Gy
    Ct[:, 1:] += Gx[:, :-1]
    Ct[1:] += Gy[:-1]
    Ct = np.where(rng.random((ny, nx)) < 0.1, -Ct, Ct)
    return Ct, Gx, Gy, rng.standard_normal((ny, nx))


def _residual(Ct, Gx, Gy, b, x):
    """b - A x; a decoupled row (Ct < 0) has no couplings, and stands at b/|Ct| in
    its neighbours' rows."""
    v = np.where(Ct < 0, b / np.abs(Ct), x)
    off = np.zeros_like(x)
    off[:, :-1] += Gx[:, :-1] * v[:, 1:]
    off[:, 1:] += Gx[:, :-1] * v[:, :-1]
    off[:-1] += Gy[:-1] * v[1:]
    off[1:] += Gy[:-1] * v[:-1]
    return b - np.abs(Ct) * x + np.where(Ct < 0, 0.0, off)


@pytest.mark.parametrize("nx,ny", [
    (1, 1), (3, 2), (63, 15), (64, 16), (65, 17),
    (64, 16 * TILE), (64, 16 * TILE + 1),      # one cluster, and groups of eight
    (64, 112 * TILE), (64, 112 * TILE + 1),    # the last groups of eight, groups of four
    (64, 128 * TILE + 1),                      # past the clusters
    (64, 148 * TILE + 1), (130, 1200), (512, 512),  # taller tiles
    (24, 10922),                               # more tiles than SMs: the general kernel
])
def test_true_residual(nx, ny):
    import torch
    sysm = _system(nx, ny)
    bufs = [torch.from_numpy(a.ravel().copy()).cuda() for a in sysm]
    for warm in (False, True):  # from zero, then from a perturbed solution
        x = torch.full((nx * ny,), np.nan, dtype=torch.float64, device="cuda") if not warm else x + 1e-3
        torch.cuda.synchronize()
        its, rel = native.cg_solve_noalloc(nx, ny, *[t.data_ptr() for t in bufs], x.data_ptr(), 1e-12, 1000,
                                           x0_from_x=warm)
        assert 0 < its < 100 and rel < 1e-12
        r = _residual(*sysm, x.cpu().numpy().reshape(ny, nx))
        assert np.linalg.norm(r) <= 1.2e-12 * np.linalg.norm(sysm[3])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(129, 33), (520, 500), (640, 610)])
def test_domain_solve_matches_the_two_phase_schedule(nx, ny, precision):
    """The same assembled system through the two-phase kernel: two solves to the same
    tolerance, compared to the solve tests' 1e-10."""
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=4, seed=41, dry_frac=0.25))
    want = native.domain_from_deck(d, schedule=native.CG_TWO_PHASE)
    prec = native.PRECISION_MIXED if precision == "mixed" else native.PRECISION_FP64
    got = native.domain_from_deck(d, precision=prec)
    for g in (want, got):
        g.phase(native.PHASE_EXPLICIT, 1)
        g.phase(native.PHASE_SOLVE, 1)
    assert max_rel(got.solution(), want.solution()) <= 1e-10


@pytest.mark.parametrize("cells_per_cta", [1, 2000, 1e9])
def test_batched_solve_whatever_the_tiles(cells_per_cta):
    """Uneven basins whose groups share CTAs: the same alone and in the mix, and with
    cells_per_cta = 1 the single-domain doubles (clusters of one solve, L2 of the other)."""
    decks = [D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=6, seed=50 + k, dry_frac=0.2))
             for k, (nx, ny) in enumerate([(200, 300), (70, 40), (64, 64), (140, 150), (33, 500)])]

    def run(ds):
        b = native.Batch(8 << 30, cells_per_cta)
        doms = [native.domain_from_deck(d) for d in ds]
        slots = [b.admit(g, 1) for g in doms]
        for _ in range(4):
            b.step()
        for s in slots:
            b.release(s)
        out = [g.download(["surf", "uuXP", "vvYP", "S"]) for g in doms]
        b.close()
        return out
    mix = run(decks)
    for k, d in enumerate(decks):
        if cells_per_cta == 1:
            g = native.domain_from_deck(d)
            assert g.run(1, 4) == 0
            alone = g.download(["surf", "uuXP", "vvYP", "S"])
        else:
            alone = run([d])[0]
        for f in alone:
            assert np.array_equal(mix[k][f], alone[f]), (k, f)

"""The streaming single-sweep solve (csrc/cg1.cu) on its own: domains past the on-chip
limit of 148 tiles of 64 x 64 cells, thin ones (24 x 10922 is 171 of them, 16384 x 16
256) and a square one, which the schedule tests at small sizes no longer reach."""
import numpy as np
import pytest

from frehdc_b200 import autotune
from frehdc_b200 import deck as D
from frehdc_b200 import native
from tests.helpers import max_rel

pytestmark = pytest.mark.gpu

SIZES = [(24, 10922), (16384, 16), (810, 790)]
FIELDS = ["surf", "uuXP", "vvYP", "S"]
PRECISIONS = {"fp64": native.PRECISION_FP64, "mixed": native.PRECISION_MIXED}


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if native.device_count() < 1:
        pytest.fail("no CUDA device visible: the GPU tests need a B200")


def _deck(nx, ny, **kw):
    return D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=8, seed=61, dry_frac=0.25, **kw))


def _solution(d, **kw):
    g = native.domain_from_deck(d, **kw)
    g.phase(native.PHASE_EXPLICIT, 1)
    g.phase(native.PHASE_SOLVE, 1)
    return g


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_matches_the_two_phase_schedule(nx, ny, precision):
    """The same assembled system through the two-phase kernel, to the solve tests' 1e-10."""
    assert not autotune.fits_on_chip(nx, ny)
    d = _deck(nx, ny)
    want = _solution(d, schedule=native.CG_TWO_PHASE)
    got = _solution(d, precision=PRECISIONS[precision])
    assert max_rel(got.solution(), want.solution()) <= 1e-10


@pytest.mark.parametrize("iters", [1, 2, 7, 8])
def test_sweeps_in_either_direction(iters):
    """Every other sweep takes the tiles in reverse: solves cut off after an odd and an
    even number of iterations against the two-phase kernel's.  Both run the same
    recurrence; eight iterations spread the roundings by far less than 1e-10."""
    d = _deck(810, 790, max_iter=iters)
    want = _solution(d, schedule=native.CG_TWO_PHASE)
    got = _solution(d)
    assert max_rel(got.solution(), want.solution()) <= 1e-10


@pytest.mark.parametrize("nx,ny", [(16384, 16), (9700, 60)])
def test_a_stalled_solve_falls_back(nx, ny):
    """A fully wet basin, wide enough that its tidal row stalls the assembled system's CG
    (as in the schedule tests): the solve starts again with that row eliminated and ends
    with the eliminated system's solution."""
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=8, seed=3))
    assert not autotune.fits_on_chip(nx, ny)
    g, e = _solution(d), _solution(d, decoupled=native.DECOUPLED_ELIMINATED)
    for h in (g, e):
        h.phase(native.PHASE_UPDATE, 1)
    st, se = g.stats(), e.stats()
    assert st["cg_fallback"] == 1 and se["cg_fallback"] == 0
    assert st["cg_rel_residual"] < d.spec.eps and st["cg_iters"] > 400
    assert max_rel(g.solution(), e.solution()) < 1e-12


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", SIZES[:2])
def test_a_wait_that_runs_out(nx, ny, precision):
    """As test_failure.py's, in the streaming kernel: the step reports the timeout, and
    after a new state the domain steps as a fresh one."""
    d = _deck(nx, ny)
    g, fresh = (native.domain_from_deck(d, precision=PRECISIONS[precision]) for _ in range(2))
    for _ in range(5):
        g.set_wait_test(1_000_000, skip_barrier_rank=0)
        with pytest.raises(native.FrehdError) as e:
            g.step(1)
        assert e.value.status == 7  # FREHD_ERR_TIMEOUT
        g.init(d.bottom, d.bottomXP, d.bottomYP, d.surf0, None, None, d.S0)
    assert g.run(1, 3) == 0 and fresh.run(1, 3) == 0
    for f in FIELDS:
        assert np.array_equal(g.download([f])[f], fresh.download([f])[f]), f

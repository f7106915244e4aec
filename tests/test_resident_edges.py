"""The resident solve (csrc/cg_res.cuh) on systems that a time step does not assemble.

Systems are diagonally dominant with smallest eigenvalue 1, as in
test_resident_solve.py, whose bound on the true residual (the recursive one,
1e-12 ||b||, and the recursion's rounding) holds for them too.
"""
import numpy as np
import pytest

from frehdc_b200 import native
from tests.test_resident_solve import _residual

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if native.device_count() < 1:
        pytest.fail("no CUDA device visible: the GPU tests need a B200")


def _solve(system, eps=1e-12, max_iter=1000, x0=None):
    import torch
    ny, nx = system[0].shape
    bufs = [torch.from_numpy(a.ravel().copy()).cuda() for a in system]
    x = torch.zeros(nx * ny, dtype=torch.float64, device="cuda") if x0 is None else \
        torch.from_numpy(x0.ravel().copy()).cuda()
    torch.cuda.synchronize()
    its, rel = native.cg_solve_noalloc(nx, ny, *[t.data_ptr() for t in bufs], x.data_ptr(), eps, max_iter,
                                       x0_from_x=x0 is not None)
    return x.cpu().numpy().reshape(ny, nx), its, rel


def _signed_system(nx, ny):
    """Couplings of both signs; Ct is 1 plus the sum of their magnitudes."""
    rng = np.random.default_rng([nx, ny, 1])
    Gx, Gy = rng.uniform(-1, 1, (ny, nx)), rng.uniform(-1, 1, (ny, nx))
    Gx[:, -1] = 0
    Gy[-1] = 0
    Ct = 1 + np.abs(Gx) + np.abs(Gy)
    Ct[:, 1:] += np.abs(Gx[:, :-1])
    Ct[1:] += np.abs(Gy[:-1])
    return np.where(rng.random((ny, nx)) < 0.1, -Ct, Ct), Gx, Gy, rng.standard_normal((ny, nx))


@pytest.mark.parametrize("nx,ny", [(3, 2), (65, 17), (130, 1200), (512, 512), (24, 10922)])
def test_couplings_of_both_signs(nx, ny):
    system = _signed_system(nx, ny)
    x, its, rel = _solve(system)
    assert 0 < its < 100 and rel < 1e-12
    assert np.linalg.norm(_residual(*system, x)) <= 1.2e-12 * np.linalg.norm(system[3])


def test_a_tolerance_no_residual_meets():
    """eps <= 0 in a domain's configuration: the solve stops at maxIter, a warning."""
    from frehdc_b200 import deck as D
    d = D.make_deck(D.DeckSpec(nx=70, ny=40, steps=4, seed=6))
    for eps in (0.0, -1e-12):
        cfg = dict(D.config_dict(d), eps=eps, maxIter=5)
        g = native.Domain(cfg, 0)
        g.set_fine_bottoms(d.zf, d.r)
        g.set_tide(D.tide_series(d))
        g.init(d.bottom, d.bottomXP, d.bottomYP, d.surf0, None, None, d.S0)
        assert g.step(1) == 5  # FREHD_ERR_CG_NOCONVERGE
        assert g.stats()["cg_iters"] == 5 and g.stats()["cg_noconverge"] == 1


@pytest.mark.parametrize("nx,ny,skip", [(48, 40, 2), (300, 60, 19), (300, 300, 94)])
def test_waits_that_run_out_while_other_ctas_start(nx, ny, skip):
    """The shortest waits, so that CTAs give up and fail the step while others of the
    same solve still read its status: every such step ends with the timeout's status,
    and after a new state the domain steps as a fresh one."""
    from frehdc_b200 import deck as D
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=40, seed=8, dry_frac=0.2))
    init = (d.bottom, d.bottomXP, d.bottomYP, d.surf0, None, None, d.S0)
    g, fresh = native.domain_from_deck(d), native.domain_from_deck(d)
    for _ in range(30):
        g.set_wait_test(1, skip_barrier_rank=skip)
        with pytest.raises(native.FrehdError) as e:
            g.step(1)
        assert e.value.status == 7  # FREHD_ERR_TIMEOUT
        g.init(*init)
    assert g.run(1, 3) == 0 and fresh.run(1, 3) == 0
    for f in ("surf", "uuXP", "vvYP", "S"):
        assert np.array_equal(g.download([f])[f], fresh.download([f])[f]), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(48, 40), (130, 500), (520, 500)])
def test_launched_without_its_clusters(nx, ny, precision):
    """A launch that does not form the clusters its kernel is told of (one cluster,
    groups of eight, tall tiles): everything goes through L2, with the same doubles."""
    from frehdc_b200 import deck as D
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=8, seed=12, dry_frac=0.2))
    prec = native.PRECISION_MIXED if precision == "mixed" else native.PRECISION_FP64
    out = []
    for plain in (False, True):
        g = native.domain_from_deck(d, precision=prec)
        g.set_solve_test(plain_launch=plain)
        assert g.run(1, 4) == 0
        out.append(g.download(["surf", "uuXP", "vvYP", "S"]))
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.parametrize("nx,ny", [(64, 250), (130, 900), (500, 540)])
def test_refinements_read_their_neighbours_new_x(nx, ny):
    """A tight tolerance, so that x passes between the tiles several times: the same
    doubles in every run, and the FP64 solution within the refinement's own bound."""
    from frehdc_b200 import deck as D
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=4, seed=33, dry_frac=0.2, eps=1e-13))

    def solution(precision, eps_inner):
        g = native.domain_from_deck(d, precision=precision, eps_inner=eps_inner)
        g.phase(native.PHASE_EXPLICIT, 1)
        g.phase(native.PHASE_SOLVE, 1)
        return g.solution()
    want = solution(native.PRECISION_FP64, 1e-5)
    first = solution(native.PRECISION_MIXED, 1e-3)
    assert np.max(np.abs(first - want)) <= 1e-10 * np.max(np.abs(want))  # the solve tests' bound
    for _ in range(10):
        assert np.array_equal(solution(native.PRECISION_MIXED, 1e-3), first)


@pytest.mark.parametrize("precision,eps", [("fp64", 1e-12), ("mixed", 1e-12), ("mixed", 1e-17)])
@pytest.mark.parametrize("nx,ny", [(40, 12), (300, 60), (64, 2100)])
def test_exchange_counter_starts_again(nx, ny, precision, eps):
    """The exchange counter passes the value from which a solve restarts it, in every
    step anew: one tile, clusters, and no clusters; with eps = 1e-17 the mixed solve's
    refinement stalls and its FP64 solve takes over in the same launch."""
    from frehdc_b200 import deck as D
    d = D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=16, seed=14, dry_frac=0.2, eps=eps))
    prec = native.PRECISION_MIXED if precision == "mixed" else native.PRECISION_FP64
    g, want = (native.domain_from_deck(d, precision=prec) for _ in range(2))
    for tt in range(1, 13):
        g.set_solve_test(first_tag=0xC0000000 - 5 * tt)
        assert g.step(tt) == want.step(tt) == 0
        assert g.step(tt + 12) == want.step(tt + 12) == 0  # from beyond the bound
        if eps < 1e-16:
            assert g.stats()["cg_fallback"] == 2
    for f in ("surf", "uuXP", "vvYP", "S"):
        assert np.array_equal(g.download([f])[f], want.download([f])[f]), f


@pytest.mark.parametrize("scale", [1e-158, 1e-150, 1.0, 1e140])
def test_right_hand_sides_of_any_size(scale):
    """beta = gamma / gamma_old, a quotient of two sums: with b of this size the sums
    leave the range in which 1 / gamma_old exists.  Scaling b by a power of two scales
    every number of the solve, so x scales to the last bit where the squares keep all
    theirs: the last ones are (1e-12)^2 of the first (b above 1e-130)."""
    rng = np.random.default_rng(21)
    nx, ny = 130, 70
    system = list(_signed_system(nx, ny))
    system[0] = np.abs(system[0])
    system[3] = rng.standard_normal((ny, nx))
    ref, its_ref, _ = _solve(system)
    p2 = 2.0 ** np.round(np.log2(scale))
    x, its, _ = _solve([*system[:3], system[3] * p2])
    assert np.all(np.isfinite(x)) and 0 < its
    if scale > 1e-130:
        assert its == its_ref and np.array_equal(x, ref * p2)
    else:  # the sums lose their bits on the way: a solution of a coarser solve
        assert np.linalg.norm(_residual(*system[:3], system[3] * p2, x) / p2) <= 1e-4 * np.linalg.norm(system[3])


@pytest.mark.parametrize("nx,ny", [(3, 2), (130, 70), (512, 512)])
def test_a_start_that_meets_the_tolerance_is_returned(nx, ny):
    """No iteration, no rounding: the caller's x comes back as it was.  (Not the solve's
    own x: that one is already a quotient by sqrt|Ct|, and the scaling back exact.)"""
    system = _signed_system(nx, ny)
    x, _, _ = _solve(system)
    x *= 1 + 1e-9 * np.random.default_rng(2).uniform(0.5, 1, x.shape)
    again, its, rel = _solve(system, eps=1e-6, x0=x)
    assert its == 0 and rel < 1e-6
    assert np.array_equal(again, x)


@pytest.mark.parametrize("nx,ny", [(48, 40), (130, 500), (512, 512), (24, 10922)])
def test_queued_solve_captured_in_a_graph(nx, ny):
    """The solve queued on a capturing stream (after a first call, which sets the device
    up) and replayed on new right-hand sides: the direct call's doubles."""
    import torch
    system = _signed_system(nx, ny)
    bufs = [torch.from_numpy(a.ravel().copy()).cuda() for a in system]
    x = torch.zeros(nx * ny, dtype=torch.float64, device="cuda")
    _solve(system)
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        native.cg_solve_noalloc(nx, ny, *[t.data_ptr() for t in bufs], x.data_ptr(), 1e-12, 1000,
                                stream=torch.cuda.current_stream().cuda_stream, wait=False)
    for k in range(3):
        b = np.random.default_rng(k).standard_normal((ny, nx))
        bufs[3].copy_(torch.from_numpy(b.ravel()))
        g.replay()
        torch.cuda.synchronize()
        want, _, _ = _solve([*system[:3], b])
        assert np.array_equal(x.cpu().numpy().reshape(ny, nx), want)


def test_domains_of_several_host_threads():
    """Solves of 16, 64 and 128 CTAs in and out of clusters on streams of their own, which
    do not all fit the device at once: the doubles of each domain stepped alone."""
    import threading

    from frehdc_b200 import deck as D
    sizes = [(128, 128), (256, 256), (512, 512), (500, 520), (70, 40), (130, 500)]
    decks = [D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=60, seed=25 + k, dry_frac=0.2))
             for k, (nx, ny) in enumerate(sizes)]
    precs = [native.PRECISION_MIXED if k % 2 else native.PRECISION_FP64 for k in range(len(decks))]
    doms = [native.domain_from_deck(d, precision=p) for d, p in zip(decks, precs)]
    status = [None] * len(doms)

    def steps(k):
        status[k] = [doms[k].run(1 + 10 * n, 10) for n in range(5)]
    threads = [threading.Thread(target=steps, args=(k,)) for k in range(len(doms))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, (g, d) in enumerate(zip(doms, decks)):
        assert status[k] == [0] * 5
        alone = native.domain_from_deck(d, precision=precs[k])
        assert alone.run(1, 50) == 0
        for f in ("surf", "uuXP", "vvYP", "S"):
            assert np.array_equal(g.download([f])[f], alone.download([f])[f]), (k, f)

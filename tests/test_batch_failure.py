"""A domain that fails or takes long inside a batch leaves the others alone (the batched
resident solve, whose CTAs go from one domain's solve to the next).

Five basins of 64 tiles each share the device's 148 CTAs, and two small ones fill in.
The waits that run out are made on the host (frehd_domain_set_wait_test); nothing
faults or hangs."""
import functools

import numpy as np
import pytest

from frehdc_b200 import deck as D
from frehdc_b200 import native

pytestmark = pytest.mark.gpu

SIZES = [(500, 500), (500, 501), (502, 500), (500, 503), (504, 500), (70, 40), (60, 14)]
FIELDS = ["surf", "uuXP", "vvYP", "S"]
STATUS_NOCONV, STATUS_TIMEOUT = 5, 7


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if native.device_count() < 1:
        pytest.fail("no CUDA device visible: the GPU tests need a B200")


def _deck(k, **kw):
    return D.make_deck(D.DeckSpec(nx=SIZES[k][0], ny=SIZES[k][1], steps=6, seed=70 + k, dry_frac=0.2, **kw))


@functools.cache
def _decks():
    return tuple(_deck(k) for k in range(len(SIZES)))


@functools.cache
def _alone(precision):
    return [_run([d], 3, precision=precision)[0] for d in _decks()]


def _run(decks, steps, waits=None, precision=native.PRECISION_FP64):
    """States and statistics of the decks stepped in one batch; waits: per domain
    (limit in ns, rank that leaves early or -1)."""
    b = native.Batch(8 << 30, 1e4)
    doms = [native.domain_from_deck(d, precision=precision) for d in decks]
    for g, w in zip(doms, waits or []):
        g.set_wait_test(w[0], skip_barrier_rank=w[1])
    slots = [b.admit(g, 1) for g in doms]
    for _ in range(steps):
        b.step()
    for s in slots:
        b.release(s)
    b.close()
    return [(g.download(FIELDS), g.stats()) for g in doms]


def _same(got, want, k):
    for f in FIELDS:
        assert np.array_equal(got[0][f], want[0][f]), (k, f)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bad", [0, 2, 4, 5])
def test_a_timeout_stays_with_its_domain(bad, precision):
    """One CTA of domain `bad` leaves its solve; the partners wait 300 ms in vain.  The
    others, whose own waits end after 100 ms, get their alone results."""
    prec = native.PRECISION_MIXED if precision == "mixed" else native.PRECISION_FP64
    decks, alone = _decks(), _alone(prec)
    waits = [(100_000_000, -1)] * len(SIZES)
    waits[bad] = (300_000_000, 0)
    got = _run(decks, 3, waits, prec)
    for k in range(len(decks)):
        if k == bad:
            assert got[k][1]["status"] == STATUS_TIMEOUT
            continue
        assert got[k][1]["status"] == 0 and got[k][1]["step"] == 3
        _same(got[k], alone[k], k)


def test_a_long_solve_holds_up_nobody():
    """A tolerance that no residual meets: one basin's solve takes all of its
    100 000 iterations, far longer than the others' waits."""
    decks = list(_decks())
    decks[4] = _deck(4, eps=0.0, max_iter=100_000)  # the largest: first in every CTA's list
    got = _run(decks, 3, [(20_000_000, -1)] * len(SIZES))
    # (and those of the first attempt, which ended as stalled)
    assert got[4][1]["cg_iters"] >= 100_000 and got[4][1]["cg_noconverge"] == 1
    alone = _alone(native.PRECISION_FP64)
    for k in (0, 1, 2, 3, 5, 6):
        assert got[k][1]["status"] == 0 and got[k][1]["step"] == 3
        _same(got[k], alone[k], k)

"""On-chip or streamed solves of a batch (frehd_batch_set_resident): a mix whose domains
lie on both sides of the on-chip limit, in every packing."""
import functools

import numpy as np
import pytest

from frehdc_b200 import deck as D
from frehdc_b200 import native

pytestmark = pytest.mark.gpu

# past the on-chip limit by tiles (171 of 64 x 64), and by cells; then ones that fit
SIZES = [(24, 10922), (800, 800), (130, 300), (64, 64), (70, 40)]
FIELDS = ["surf", "uuXP", "vvYP", "S"]


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if native.device_count() < 1:
        pytest.fail("no CUDA device visible: the GPU tests need a B200")


@functools.cache
def _decks():
    return [D.make_deck(D.DeckSpec(nx=nx, ny=ny, steps=2100, seed=90 + k, dry_frac=0.2))
            for k, (nx, ny) in enumerate(SIZES)]


def _run(decks, packing, precision, steps=3):
    b = native.Batch(16 << 30, 20000)
    b.set_cg_packing(packing)
    doms = [native.domain_from_deck(d, precision=precision) for d in decks]
    slots = [b.admit(g, 1) for g in doms]
    for _ in range(steps):
        b.step()
    for s in slots:
        b.release(s)
    b.close()
    return [g.download(FIELDS) for g in doms]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("packing", ["tile_list", "cta_groups", "cta_groups_streamed"])
def test_both_sides_of_the_limit(packing, precision):
    """The same alone and in the mix, and the two-phase solve's states to the parity
    tests' 1e-9 of the surface, and the velocities' that follows from it (three steps
    from rest hardly move any water: a bound by the velocities themselves means nothing)."""
    from frehdc_b200 import autotune
    prec = native.PRECISION_MIXED if precision == "mixed" else native.PRECISION_FP64
    mix = _run(_decks(), autotune.PACKINGS[packing], prec)
    for k, d in enumerate(_decks()):
        alone = _run([d], autotune.PACKINGS[packing], prec)[0]
        want = native.domain_from_deck(d, schedule=native.CG_TWO_PHASE)
        assert want.run(1, 3) == 0
        ref = want.download(FIELDS)
        for f in FIELDS:
            assert np.array_equal(mix[k][f], alone[f]), (k, f)
            # (a face velocity moves by g dt/dx times the difference of two surfaces)
            scale = 2 * 9.81 * np.max(np.abs(ref["surf"])) * d.spec.dt / d.spec.dx if f in ("uuXP", "vvYP") \
                else np.max(np.abs(ref[f]))
            assert np.max(np.abs(mix[k][f] - ref[f])) <= 1e-9 * scale, (k, f)


def test_a_server_streams_when_told():
    """frehd_server_set_resident: the batch's streamed doubles; refused while the server
    holds a request."""
    d = _decks()[2]
    want = _run([d], native.BATCH_CTA_GROUPS_STREAMED, native.PRECISION_FP64)[0]
    srv = native.Server(16 << 30, 20000)
    srv.set_resident(False)
    g, late = native.domain_from_deck(d), native.domain_from_deck(d)
    srv.submit(g, 3)
    srv.submit(late, 2000)
    with pytest.raises(native.FrehdError) as e:
        srv.set_resident(True)
    assert e.value.status == 8  # FREHD_ERR_STATE
    done = []
    while len(done) < 2:
        done += srv.poll(timeout_ms=200)
    srv.close()
    assert {r["status"] for r in done} == {0}
    got = g.download(FIELDS)
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f

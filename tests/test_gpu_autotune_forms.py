"""The autotuner and the two forms of the transport.

- Widths are reported as they are in use: 120 for a small batch that nothing has
  tuned (the narrow form), 192 for a large one.
- What was tuned in a small batch stays with small batches, and the other way
  round.
- In a large batch every candidate is the wide form: a tuned batch whose classes
  took other widths than the default gives the bits of an untuned one."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Batch
from tests.helpers import small
from tests.test_gpu_autotune import CAND, _batch

pytestmark = pytest.mark.gpu


def _disks(sizes, **over):
    PL = [small(kind, nrad, nsec, **over)[:2] for kind, nrad, nsec in sizes]
    return [p for p, _ in PL], [q for _, q in PL]


# sector counts that no other test tunes
def test_reported_and_kept_by_form(gpu):
    few, many = [("iso", 64, 516)], [("iso", 64, 516)] * 10  # 40 and 400 items of 120 sectors
    a, b = Batch(*_disks(few)), Batch(*_disks(many))
    assert a.segments() == [120]
    assert b.segments() == [192] * 10
    seg = a.autotune(reps=2)
    assert a.segments() == [seg] and seg == 96  # 48 items of 96 sectors
    assert Batch(*_disks(few)).segments() == [seg]
    assert Batch(*_disks(many)).segments() == [192] * 10
    seg = b.autotune(reps=2)
    assert b.segments() == [seg] * 10 and seg in CAND
    assert Batch(*_disks(many)).segments() == [seg] * 10
    assert Batch(*_disks(few)).segments() == a.segments()


def test_narrow_items_stay_two_per_sm(gpu):
    # 240 items of 120 sectors, 320 of 96; the width that a smaller batch of the class took
    # is not taken over
    few = Batch(*_disks([("iso", 64, 700)]))
    assert few.autotune(reps=2) == 96
    b = Batch(*_disks([("iso", 320, 700)]))
    assert b.segments() == [120]
    assert b.autotune(reps=2) == 120 and b.segments() == [120]


def test_wide_widths_keep_results(gpu):
    # 244 sectors: two segments at the default width, one at 244
    P, L = _disks([("iso", 400, 244), ("adi", 400, 244), ("iso", 401, 452), ("adi", 200, 676), ("iso", 400, 244)],
                  DT="0.02")
    tuned, plain = _batch(P, L), _batch(P, L)
    assert plain.segments() == [192] * 5
    tuned.autotune(reps=3)
    segs = tuned.segments()
    print("\nwide widths per disk:", segs)
    assert set(segs) <= CAND and segs[0] == segs[4]
    assert any(s != 192 for s in segs)
    for b in (tuned, plain):
        b.advance(2)
    for k in range(len(P)):
        a, c = tuned.fields(k), plain.fields(k)
        for f in a:
            assert np.array_equal(a[f], c[f]), (k, f)

"""Order of the rrule forward's launches on its two streams, on a CUDA runtime without a
device: the coefficients of a forward are not rewritten while the pullback records of an
earlier one, which only its pullback waits for, may still be read from them."""
import pytest

import fakecuda

CALLS = """
h = plan([0, 1, 2], 3, 2, int(sys.argv[3]), 200)
ops()
def rrule():
    assert L.aok_overlap2c_rrule(h, *[P(A)] * 7, I64(200), F64(1.0), P(0x77)) == 0
def pull():
    assert L.aok_overlap_pullback_ps_rrule(h, *[P(A)] * 9, I64(200), F64(1.0), P(0x77)) == 0
def whole():
    assert L.aok_overlap_pullback_ps(h, *[P(A)] * 9, I64(200), F64(1.0), P(0x77)) == 0
for f in (rrule, rrule, rrule, rrule, pull, rrule, pull, rrule, whole, rrule, rrule, whole, whole, rrule, pull):
    f()
print(json.dumps(ops()))
"""


@pytest.mark.parametrize("prec", [0, 1])
def test_coefficients_are_not_rewritten_under_the_records(tmp_path, prec):
    log = fakecuda.run(CALLS.replace("int(sys.argv[3])", str(prec)), tmp_path)
    launches = [(k, table) for k, _, table in log if k.startswith("launch:")]
    writes = [(i, t) for i, (k, t) in enumerate(launches) if "k_compile_coefI" in k]
    reads = [(i, t) for i, (k, t) in enumerate(launches) if "k_prep_pbI" in k]
    assert len(writes) == len(reads) == 12
    pairs = 0
    for w, table in writes:
        for r, of in reads:
            if of == table and r < w:
                assert fakecuda.ordered(log, r, w), (r, w)
                pairs += 1
            if of == table and r > w:
                assert fakecuda.ordered(log, w, r), (w, r)
    assert pairs

"""Set-up of the 3-center overlap when device memory runs out, on a CUDA runtime without a
device: a failed first call leaves nothing behind, and the next one starts again."""
import pytest

import fakecuda

FIRST_CALL = """
def call(h):
    return L.aok_overlap3c(h, P(A), P(A), P(A), P(A), P(A), P(A), P(A), P(A), P(A), I64(40), F64(1.0), P(0x77))
def kernels():
    return [k[0] for k in ops() if k[0].startswith("launch:")]
out = []
for ls, K, prec in (([0, 1, 2, 3], 2, 0), ([0, 1, 2, 3], 2, 1), ([0, 1], 2, 0)):
    h = plan(ls, K, 2, prec, 100)
    base = fake.fake_live()
    fake.fake_fail(*NEVER)
    assert call(h) == 0
    want, full = kernels(), fake.fake_live()
    L.aok_plan_destroy(h)
    at = 0
    while True:                                    # allocation `at` of the first call fails
        h = plan(ls, K, 2, prec, 100)
        ops()
        fake.fake_fail(at, NEVER[1])
        failed = call(h)
        after, got = fake.fake_live(), kernels()
        fake.fake_fail(*NEVER)
        again = call(h)
        out.append(dict(ls=len(ls), prec=prec, at=at, failed=failed, got=got, left=after - base, again=again,
                        kept=fake.fake_live() - full, same=kernels() == want))
        L.aok_plan_destroy(h)
        at += 1
        if at > full - base:                       # every allocation of the call has failed once
            break
print(json.dumps(dict(out=out, live=fake.fake_live(), bad=fake.fake_bad_frees())))
"""


def test_failed_allocation_leaves_nothing_behind(tmp_path):
    r = fakecuda.run(FIRST_CALL, tmp_path)
    assert r["live"] == 0 and r["bad"] == 0
    assert any(c["failed"] for c in r["out"])
    for c in r["out"]:
        if c["failed"]:
            assert not c["got"], c                 # nothing launched
            assert c["again"] == 0 and c["kept"] == 0 and c["same"], c


NO_ROOM = """
out = []
for prec in (0, 1):
    for gb in (False, True):
        h = plan([0, 1, 2, 3], 3, 1 if gb else 2, prec, 5000)
        base = fake.fake_live()
        if WHAT == "buffer":
            fake.fake_fail(-1, 1 << 20)            # the moments want more than that
        else:
            fake.fake_fail_kernel(b"k_transform3") # no local memory for its routines
        for repeat in range(2):
            ops()
            if gb:
                st = L.aok_overlap3c_gb(h, *[P(A)] * 8, I64(5000), P(0x77))
            else:
                st = L.aok_overlap3c(h, *[P(A)] * 9, I64(5000), F64(1.0), P(0x77))
            out.append(dict(st=st, k=[k[0] for k in ops() if k[0].startswith("launch:")],
                            n=fake.fake_live() - base))
        fake.fake_fail(*NEVER)
        L.aok_plan_destroy(h)
print(json.dumps(dict(out=out, live=fake.fake_live(), bad=fake.fake_bad_frees())))
"""


@pytest.mark.parametrize("what", ["buffer", "local memory"])
def test_without_room_for_moments_the_tables_serve(tmp_path, what):
    r = fakecuda.run(f"WHAT = {what!r}" + NO_ROOM, tmp_path)
    assert r["live"] == 0 and r["bad"] == 0
    assert len(r["out"]) == 8 and len({c["n"] for c in r["out"]}) == 1
    for c in r["out"]:
        assert c["st"] == 0, c
        assert sum("k_overlap3c" in k for k in c["k"]) == 1
        assert not any("moments3" in k or "transform3" in k or "prepm3" in k for k in c["k"]), c

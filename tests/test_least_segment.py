"""Lone ranges on both sides of the rule for the least segment, against the
oracle, by the one-call path and as launch plans (which sieve a segment in one
CTA each)."""
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("count", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2", "max_gap", "max_gap_start", "num_gaps")


# sieving primes times segments of 4 KiB, per SM: about 2300 and 2900 at each end
@pytest.mark.parametrize("b,widths", [(10**9 + 1, (245730, 245760, 245790, 12 * 10**6, 16 * 10**6)),
                                      (3 * 10**9, (5 * 10**5, 75 * 10**5, 10**7)),
                                      (10**10, (10**6 + 1, 45 * 10**5, 58 * 10**5)),
                                      (10**11, (2 * 10**6, 15 * 10**5, 19 * 10**5 + 7)),
                                      (10**12, (5 * 10**5, 491521, 7 * 10**5))])
def test_both_sides(vg, oracle_lib, b, widths):
    from voss_gb300.plan import SievePlan
    for w in widths:
        orc = oracle_lib.range_stats(b - w, b)
        plan = SievePlan([(b - w, b)])
        plan.launch(0)
        for st in (vg.range_stats(b - w, b, full=True), plan.results(0)[0]):
            assert [getattr(st, k) for k in KEYS] == [orc[k] for k in KEYS], (b, w)
            assert (st.first_prime, st.last_prime) == (orc["first"], orc["last"]), (b, w)
            assert st.gap_hist[:201] == [int(x) for x in orc["hist"][:201]], (b, w)
        plan.close()

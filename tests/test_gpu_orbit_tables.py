"""Perturbation frames on orbits whose lengths lie around the table kernel's blocks (64 threads) and the composed
blocks (16 and 64 steps, which need an orbit longer than that), against the multi-word oracle.  The bars are those of
the shallow views in test_gpu_perturb.py."""
import pytest

pytestmark = pytest.mark.gpu

from tests.test_gpu_perturb import hp_counts, perturb_frame  # noqa: E402


@pytest.mark.parametrize("max_iter", [1, 2, 15, 16, 17, 18, 63, 64, 65, 66, 81, 128, 129, 1000])
def test_orbit_lengths(cuda, oracle, max_iter):
    from fractions import Fraction

    import chaos_gb300 as cg
    w, h, bits, ps = 48, 32, 192, 2e-3 / 48
    centre = (cg.to_hex_fixed(Fraction(-0.7455), bits), cg.to_hex_fixed(Fraction(0.1133), bits))
    orbit = cg.Orbit(*centre, bits, max_iter)
    assert orbit.info()["stored"] <= max_iter + 1
    want = hp_counts(oracle, centre, w, h, 1, 0, 0, ps, bits, max_iter)
    for tier, bar in ((cg.TIER_PERTURB_F64, 0.005), (cg.TIER_PERTURB_F32, 0.01)):
        if tier == cg.TIER_PERTURB_F32 and max_iter > 129:
            continue  # binary32 differences that rebase on this early escaping orbit lose 5 % of the counts by 1000
        got, _, _ = perturb_frame(cuda, orbit, w, h, max_iter, 1, cg.SAMPLES_CENTER, tier, ps, seed=0)
        assert float((got != want).mean()) <= bar, tier


def test_far_offsets_stay_tested_in_full(cuda, oracle):
    """Pixels so large that a binary64 difference leaves the binary32 range: every sample escapes at once."""
    import chaos_gb300 as cg
    orbit = cg.Orbit("0.0", "1.0", 128, 100)
    got, _, _ = perturb_frame(cuda, orbit, 9, 7, 100, 1, cg.SAMPLES_JITTER, cg.TIER_PERTURB_F64, 1e40)
    assert (got == 1).all()

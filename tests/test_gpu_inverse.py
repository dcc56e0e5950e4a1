"""Device forms of the field inverse and of point sums by four lanes."""
import pytest

pytestmark = pytest.mark.gpu


def test_inverse_and_quad_sums(gpu_pkg):
    """Inverses of 0, powers of two and their negatives and random values, by one
    lane and by four; sums by quads with equal, opposite and infinite points in
    some quads of a warp, all points with denominators of their own."""
    fails = gpu_pkg.selftest()
    for check in ("fq_inverse", "fr_inverse", "fq_inverse_quad", "quad_add", "quad_dbl"):
        assert fails[check] == 0, fails

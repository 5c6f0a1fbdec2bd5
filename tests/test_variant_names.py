"""Report names of the kernel variants (CPU, no GPU): every current and every
earlier name resolves, others are refused."""
import pytest


def test_names_resolve(pkg):
    for p, pname in pkg.PASS_NAMES.items():
        for v, name in pkg.VARIANT_NAMES[p].items():
            assert pkg.variant_by_name(pname, name) == (p, v)
    for name, v in (("ring_3x12k", 0), ("ring_3x12k_evict_first", 1), ("ring_2x8k_evict_first", 2),
                    ("ring_3x8k_evict_first", 3)):
        assert pkg.variant_by_name("y2_solve", name) == (pkg.PASS_Y2, v)
    for bad in (("y2_solve", "ring_9x9k"), ("x_pass", "block_fft")):
        with pytest.raises(KeyError):
            pkg.variant_by_name(*bad)

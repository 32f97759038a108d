"""ws_matcher_info.last_launches counts every kernel that a scan enqueues."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regexes,kernels", [
    ([], 3),                    # counters, filter, verify
    (["key=[0-9]{1,3}"], 7),    # and the walk and reverse walks behind the filter, scatter, resolution
])
def test_last_launches_is_the_number_of_kernels(regexes, kernels):
    import warpstate_b200 as ws
    b = ws.PatternSet.builder().literal_bytes(b"needle").literal_bytes(b"haystack")
    for r in regexes:
        b = b.regex(r)
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig())
    for _ in range(2):
        assert len(m.scan_array(b"." * 5000 + b"needle")) == 1
        assert m.info()["last_launches"] == kernels

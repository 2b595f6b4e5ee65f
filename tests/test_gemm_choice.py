"""Which kernel a plain product takes (a rule on its sizes, evaluated on the host)."""
import pytest


@pytest.fixture(scope="module")
def choice():
    from ps_lite_b200 import _lib
    return _lib.device_lib().psdev_gemm_choice


def _ctas(code, m, n):
    return -(-m // 128) * -(-n // (code % 1000)) * (code // 1000)


@pytest.mark.parametrize("m", [1, 8, 16, 63, 64, 100, 128, 200, 255, 256, 300, 511, 1024, 2048])
@pytest.mark.parametrize("n,k", [(8192, 1024), (32768, 1024), (50264, 1024), (65536, 512),
                                 (16384, 4096), (16384, 16384), (128, 65536), (4104, 4096)])
def test_small_tiles_outside_of_the_measured_sizes(choice, m, n, k):
    """No more of them than fit on the GPU, whatever the fitted times say."""
    code = choice(m, n, k)
    if 1000 <= code < 2000 and (m < 64 or n * k > 4096 * 4096):
        assert _ctas(code, m, n) <= (148 if m < 64 else 444 if m <= 128 else 296)
    elif code >= 2000 and code not in (2256, 2512):
        assert _ctas(code, m, n) <= 296


@pytest.mark.parametrize("m,n,k,code", [(300, 16384, 4096, 2512), (1, 50264, 1024, 0), (64, 50264, 1024, 1128),
                                        (1024, 1024, 1024, 1064), (7572, 288, 256, 1064),
                                        (16384, 3072, 1024, 2512), (64, 256, 4096, 8064)])
def test_choices(choice, m, n, k, code):
    assert choice(m, n, k) == code


@pytest.mark.parametrize("m,n,k", [(3013, 1616, 2104), (1603, 1624, 824), (7525, 280, 3528),
                                   (6319, 672, 2648), (301, 3248, 2136)])
def test_rows_that_begin_inside_a_sector(choice, m, n, k):
    """Pairs, where small tiles would read such rows."""
    assert choice(m, n, k) in (2256, 2512)


@pytest.mark.parametrize("m,n", [(1, 256), (64, 64), (64, 256), (100, 200), (128, 256), (128, 512), (256, 256)])
def test_a_longer_k_keeps_its_parts(choice, m, n):
    """A few tiles: one more k-block does not take CTAs from the cluster that shares it.  (From 32
    k-blocks on: of fewer, 17 say, a part of eight has as many as one of six would, and a cluster of
    four can be ahead.)"""
    parts = [choice(m, n, k) // 1000 for k in range(2048, 16385, 64)]
    assert all(b >= a for a, b in zip(parts, parts[1:])) and parts[-1] == 8

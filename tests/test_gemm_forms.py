"""Which form of the GEMM kernel a product takes: the host's cost model, without a GPU, for a device with the residency of
148 SMs (74 clusters of two CTAs, 33 of four)."""
import pytest

from jaxpp_b200.ops import native

PAIR256, PAIR128, ONE256, ONE128, ONE64 = range(5)
TILE = {PAIR256: (256, 256), PAIR128: (256, 128), ONE256: (128, 256), ONE128: (128, 128), ONE64: (128, 64)}
CTAS, PAIRS, QUADS = 148, 74, 33


def choice(M, N, K, batch=1, counted=False, out_fp32=False):
    r = native.load().jpb_gemm_form(batch, M, N, K, int(out_fp32), int(counted), CTAS, PAIRS, QUADS)
    return r % 16, r // 16


def tiles(form, M, N, batch=1):
    m, n = TILE[form]
    return batch * -(-M // m) * -(-N // n)


@pytest.mark.parametrize("K", [512, 1024, 4096, 8192, 11008, 28672])
def test_divided_reductions_run_in_one_round(K):
    """All parts of a tile wait for one another in a cluster; clusters that are not resident make a second round, which is
    longer than the undivided product."""
    divided = set()
    for M in (8, 77, 128, 200, 256, 512):
        for N in range(64, 6000, 64):
            form, split = choice(M, N, K)
            if split > 1:
                assert form == ONE64 and tiles(form, M, N) <= {2: PAIRS, 4: QUADS}[split], (M, N, K)
                divided.add(split)
            assert choice(M, N, K, counted=True)[1] == 1
    assert K < 4096 or divided == {2, 4}


@pytest.mark.parametrize("M,N,K", [(77, 22016, 4096), (128, 22016, 4096), (8, 32000, 4096), (128, 28672, 1024), (384, 11008, 4096)])
def test_wide_products_of_few_rows_take_one_round(M, N, K):
    form, split = choice(M, N, K)
    assert split == 1 and tiles(form, M, N) <= (CTAS if form >= ONE256 else PAIRS)


def test_large_products_take_pairs():
    for M, N, K in ((4096, 4096, 4096), (4096, 12288, 4096), (4096, 32000, 4096), (16384, 4096, 11008), (8192, 28672, 8192)):
        assert choice(M, N, K) == (PAIR256, 1)

"""The sums of a product do not depend on the tile the chooser takes: every width adds in the same order. The number of shares a contraction is
cut into does decide that order; products that ask for it (an LSTM's) get a fixed function of the extents."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _err():
    return torch.zeros(1, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(512, 384, 1000, False, False), (520, 392, 72, False, True), (304, 264, 2056, True, True)])
def test_every_width_gives_the_same_bits(M, N, K, a_mn, b_mn):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(M)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda").bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda").bfloat16()
    for split in (1, 3) if K > 192 else (1,):
        outs = []
        for bn in (64, 128, 256) + ((192, 512) if split == 1 else ()):
            c = torch.empty(M, N, device="cuda")
            if split == 1:
                E.gemm(a, b, c, a_mn, b_mn, 0, None, None, None, 1.0, 0.0, _err(), bn)
            else:
                E.gemm_split(a, b, c, a_mn, b_mn, 0, None, None, None, 1.0, 0.0, _err(), bn, split)
            outs.append(c)
        assert all(torch.equal(outs[0], c) for c in outs[1:])


# the recurrence of an LSTM of 2048 cells, its weight gradients, the products with sampled classes, and a long contraction
@pytest.mark.parametrize("M,N,K,mn,shares", [(128, 8192, 1024, False, 1), (128, 512, 2048, False, 8), (128, 2048, 512, False, 1),
                                             (128, 1024, 8192, False, 8), (512, 2048, 2560, True, 4), (2560, 512, 8192, False, 3),
                                             (8192, 512, 2560, True, 1), (256, 256, 16384, False, 8)])
def test_shares_of_a_contraction(M, N, K, mn, shares):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the counts below are for 148 SMs")
    bn, split = E.gemm_choice(M, N, K, 1, 0, mn, True, True)
    assert split == shares
    torch.manual_seed(K)
    a = torch.randn((K, M) if mn else (M, K), device="cuda").bfloat16()
    b = torch.randn((K, N) if mn else (N, K), device="cuda").bfloat16()
    got, want = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    E.gemm(a, b, got, mn, mn, 0, None, None, None, 1.0, 0.0, _err(), -1)
    if shares > 1:
        E.gemm_split(a, b, want, mn, mn, 0, None, None, None, 1.0, 0.0, _err(), bn, shares)
    else:
        E.gemm(a, b, want, mn, mn, 0, None, None, None, 1.0, 0.0, _err(), 64)
    assert torch.equal(got, want)


def test_long_contractions_over_rows_off_their_lines():
    """Operands whose rows do not start on 128-byte lines cost more to fetch: wide tiles and many shares."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the counts below are for 148 SMs")
    assert E.gemm_choice(88, 3512, 31296, 1, 0, True) == (256, 8)
    assert E.gemm_choice(2144, 176, 17480, 1, 2, False) == (256, 6)
    assert E.gemm_choice(2376, 968, 5520, 1, 1, False) == (512, 1)
    assert E.gemm_choice(1592, 1640, 12072, 1, 0, False) == (512, 1)
    for M, N, K in ((176, 5456, 3912), (3072, 1024, 4096), (232, 232, 5512)):
        torch.manual_seed(M)
        a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
        bn, split = E.gemm_choice(M, N, K, 1, 0, False, True)
        got, want = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
        E.gemm(a, b, got, False, False, 0, None, None, None, 1.0, 0.0, _err(), 0)
        if split > 1:
            E.gemm_split(a, b, want, False, False, 0, None, None, None, 1.0, 0.0, _err(), bn, split)
        else:
            E.gemm(a, b, want, False, False, 0, None, None, None, 1.0, 0.0, _err(), bn)
        assert torch.equal(got, want)

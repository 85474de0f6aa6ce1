"""The tcgen05 GEMMs at shapes that lead to each of their tile widths and to split K, with column counts that are no
multiple of the width and more tiles than SMs, on integers: every order of the sums gives the same fp32 value."""
import pytest

SHAPES = [(64, 64, 128), (64, 1024, 128), (130, 64, 19072), (129, 320, 18944), (257, 512, 10240), (129, 192, 18944), (129, 320, 19072),
          (129, 1024, 19072), (257, 1024, 18944), (1000, 1024, 6400), (1000, 2560, 6400), (129, 2560, 2560)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_tiles_exact_on_integers(cuda, M, K, N):
    """|a| <= 4, |w| <= 2 (weights of 8 levels times 1/4): sums below 2^24 quarters, so the fp16 result is one rounding of
    the exact sum for the fp16 and the W4A16 kernel alike."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M + 3 * K + 7 * N)
    a = torch.randint(-4, 5, (M, K), device="cuda", generator=g).half()
    q = torch.randint(0, 16, (K, N), device="cuda", generator=g, dtype=torch.uint8)
    scales = torch.full((K // 64, N), 0.25, device="cuda").half()
    w = ((q.float() - 8) * 0.25).half()
    want = (a.double() @ w.double()).half()
    slot = torch.cat([(q[:, 0::2] | q[:, 1::2] << 4).reshape(-1), scales.view(torch.uint8).reshape(-1)]).contiguous()
    packed = torch.zeros(K * N // 8, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    assert cuda.gehtp_dev_w4_repack(slot.data_ptr(), packed.data_ptr(), K, N) == 0
    runs = [lambda y: cuda.gehtp_dev_w4a16_matmul(a.data_ptr(), packed.data_ptr(), scales.data_ptr(), y.data_ptr(), M, K, N, 2)]
    if M >= 128:
        wt = w.T.contiguous()
        torch.cuda.synchronize()
        runs.append(lambda y: cuda.gehtp_dev_matmul_f16_nk(a.data_ptr(), wt.data_ptr(), y.data_ptr(), M, K, N))
    for run in runs:
        y = torch.full((M + 1, N), 7.0, device="cuda").half()          # one row more: nothing is written behind the last
        torch.cuda.synchronize()
        assert run(y) == 0, cuda.gehtp_cuda_last_error()
        assert cuda.gehtp_cuda_sync() == 0
        assert torch.equal(y[:M], want) and (y[M] == 7.0).all()

"""The surrogate's sums over pixels (bias, first layer's and head's weight
gradients) where a block takes several tiles of rows: the kernels with 16-byte
loads against the one-channel kernels, which the same call takes for a pointer,
stride or offset that is not aligned. Both add in pixel order: the same bits.
Blocks of 300 rows and more (tiles of 64 to 256), with tails, that cross image
rows and images; widths below, at and beside multiples of 8."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _call(lib, name, *args):
    import torch
    a = [ctypes.c_void_p(t.data_ptr()) if isinstance(t, torch.Tensor) else t for t in args]
    assert getattr(lib, name)(*a, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, name


def _shifted(t):
    """The same values one element off a 16-byte boundary."""
    import torch
    out = torch.zeros(t.numel() + 1, dtype=t.dtype, device=t.device)
    out[1:] = t.reshape(-1)
    return out[1:]


@pytest.mark.parametrize('C,N,H,W', [(32, 3, 173, 171), (8, 3, 173, 171), (64, 2, 211, 211), (32, 5, 149, 120),
                                     (32, 900, 10, 10), (16, 2000, 15, 3), (256, 3, 173, 171)])
def test_staged_sums_are_the_scalar_kernels(cuda_lib, C, N, H, W):
    import torch
    lib, P = cuda_lib, N * H * W
    g = torch.Generator().manual_seed(C + W)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    size = lambda w: int(lib.clv_unet_rows_scratch_bytes(w))
    z = rnd(P, C).to(torch.bfloat16)
    scratch = torch.zeros(size(9 * C) // 4 + 4, device='cuda')
    nb = ctypes.c_size_t(size(9 * C))
    # bias
    a, b = torch.zeros(C, device='cuda'), torch.zeros(C, device='cuda')
    wide = torch.zeros(P, C + 4, dtype=torch.bfloat16, device='cuda')
    wide[:, :C] = z
    _call(lib, 'clv_unet_bias_grad', z, C, ctypes.c_longlong(P), C, a, scratch, nb)
    _call(lib, 'clv_unet_bias_grad', wide, C + 4, ctypes.c_longlong(P), C, b, scratch, nb)
    assert torch.equal(a, b)
    # first layer (3 C <= 256 takes the tiles)
    img = rnd(N, H, W)
    a, b = torch.zeros(9, C, device='cuda'), torch.zeros(9, C, device='cuda')
    _call(lib, 'clv_unet_first_wgrad', img, z, N, H, W, C, a, scratch, nb)
    _call(lib, 'clv_unet_first_wgrad', img, _shifted(z), N, H, W, C, b, scratch, nb)
    assert torch.equal(a, b)
    # head
    for K in (1, 6, 8):
        go, wh = rnd(P, K), rnd(C, K)
        hs = torch.zeros(size((C + 1) * K) // 4 + 4, device='cuda')
        hb = ctypes.c_size_t(size((C + 1) * K))
        outs = []
        for y, cs in ((z, C), (wide, C + 4)):
            gz, dwb = torch.zeros_like(z), torch.zeros(C + 1, K, device='cuda')
            _call(lib, 'clv_unet_head_bwd', y, cs, 0, z, go, wh, ctypes.c_longlong(P), C, K, gz, dwb, hs, hb)
            outs.append((gz, dwb))
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1]), K
    # against 64 bits: sums of P unit products in FP32, P 2^-23 with 16 to spare
    want = z.double().sum(0)
    _call(lib, 'clv_unet_bias_grad', z, C, ctypes.c_longlong(P), C, a[0], scratch, nb)
    assert float((a[0].double() - want).abs().max()) <= 16 * P * 2.0 ** -23

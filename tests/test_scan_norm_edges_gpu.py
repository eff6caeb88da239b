"""minGRU scan with T split over a cluster, and the RMSNorm backward with several warps per row, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from gruboros_b200.ops import _lib as L
    from gruboros_b200.ops import kernels as K
    from gruboros_b200.ops import reference as R

DEV = "cuda"


def close(got, want, rtol, atol, what):
    err = (got.double() - want.double()).abs()
    assert not (err > atol + rtol * want.double().abs()).any(), (what, err.max().item())


# 64 and 128 steps per CTA and round, clusters of 2, 4 and 8: below, at and beyond one and several whole rounds
@pytest.mark.parametrize("T", [65, 127, 129, 256, 511, 513, 1024, 1025, 2049, 4097])
@pytest.mark.parametrize("B,C", [(1, 64), (2, 136)])
def test_scan_split_over_clusters(B, C, T):
    g = torch.Generator(device=DEV).manual_seed(T + C)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    ku, gr = rn(B, T, 2 * C), rn(B, T, C)
    u, k = ku[..., :C], ku[..., C:]
    h0 = torch.rand(B, C, device=DEV, generator=g) + 0.1
    h, dku = torch.full_like(gr, float("nan")), torch.full_like(ku, float("nan"))
    hl, dhl, dh0 = torch.zeros_like(h0), torch.randn(B, C, device=DEV, generator=g), torch.zeros_like(h0)
    K.scan_fwd(k, u, h, h0=h0, h_last=hl)
    kd, ud, h0d = (t.double().requires_grad_(True) for t in (k, u, h0))
    href, hlref = R.scan_ref(kd, ud, h0d)
    ((href * gr.double()).sum() + (hlref * dhl.double()).sum()).backward()
    K.scan_bwd(k, u, h, gr, dku[..., C:], dku[..., :C], h0=h0, dh_last=dhl, dh0=dh0)
    L.check_device_status()
    close(h, href.detach(), 1e-2, 1e-3, "h")                    # bf16 output (2^-8) of fp32 sums
    close(hl, hlref.detach(), 1e-4, 1e-5, "h_last")
    s = max(1.0, kd.grad.abs().max().item())
    close(dku[..., C:], kd.grad, 3e-2, 1e-2 * s, "dk")          # g - h_{t-1} cancels: the error is of h's bf16 size
    close(dku[..., :C], ud.grad, 3e-2, 1e-2 * s, "du")
    close(dh0, h0d.grad, 1e-3, 1e-3 * s, "dh0")


@pytest.mark.parametrize("D", [64, 256, 320, 512, 516, 1024, 1028, 2048, 2056, 3072, 3080, 4096, 4100])
@pytest.mark.parametrize("M", [1, 7, 1300])
def test_rmsnorm_bwd_widths(M, D):
    g = torch.Generator(device=DEV).manual_seed(D + M)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    dy, x, w, rin = rn(M, D).bfloat16(), rn(M, D), rn(D), rn(M, D)
    rstd = torch.rsqrt(x.pow(2).mean(-1) + 1e-6)
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd * dy.double()).sum().backward()
    out, out16 = torch.full_like(x, float("nan")), torch.full_like(dy, float("nan"))
    dw, dcol = torch.ones_like(w), torch.ones_like(w)
    K.rmsnorm_bwd(dy, x, rstd, w, rin, out, out16, dw, dcol)
    want = xd.grad + rin.double()
    # fp32 sums of M (columns) or D (row) terms of order one: sqrt(n) 2^-24 times their size, with room for the order
    close(out, want, 1e-4, 1e-4, "residual gradient")
    close(out16, want, 1e-2, 1e-3, "its bf16 copy")
    close(dw - 1, wd.grad, 1e-4, 2e-5 * M ** 0.5 + 1e-4, "weight gradient")
    close(dcol - 1, want.sum(0), 1e-4, 2e-5 * M ** 0.5 + 1e-4, "column sums")

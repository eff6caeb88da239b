"""Single-CTA GEMM with K split over a cluster: every epilogue, ragged edges, against fp64 products of the bf16 operands."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from gruboros_b200.ops import _lib as L
    from gruboros_b200.ops import kernels as K

DEV = "cuda"


def close(got, want, rtol, atol, what):
    err = (got.double() - want.double()).abs()
    assert not (err > atol + rtol * want.double().abs()).any(), (what, err.max().item())


@pytest.fixture(autouse=True)
def single_cta():
    old, K.GEMM_MODE = K.GEMM_MODE, "1cta"
    yield
    K.GEMM_MODE = old
    L.check_device_status()


# clusters of 1, 2, 3, 4 and 8 CTAs; k-blocks of 64 that divide evenly, leave a short last CTA, or are fewer than asked for
@pytest.mark.parametrize("S", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("M,N,Kd", [(1, 8, 64), (127, 136, 520), (130, 128, 264), (257, 264, 1000)])
def test_split_epilogues(S, M, N, Kd):
    g = torch.Generator(device=DEV).manual_seed(M + S)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x, w = rn(M, Kd).bfloat16(), (rn(N, Kd) / Kd ** 0.5).bfloat16()
    acc = x.double() @ w.double().t()
    ssq, eps = torch.rand(M, 5, device=DEV, generator=g) + 0.5, 1e-6
    rs = torch.rsqrt(ssq.double().sum(1) / Kd + eps)[:, None]
    bias, rstd = rn(N), torch.full((M,), float("nan"), device=DEV)
    nan = lambda *s, dtype=torch.bfloat16: torch.full(s, float("nan"), device=DEV, dtype=dtype)
    f32 = torch.float32
    tol = 1e-4 * rs.abs().max().item()                    # fp32 accumulation of K products of order 1 / sqrt(K)

    out = nan(M, N)
    K.gemm(0, 0, K.EPI_STORE_BF16, x, w, M, N, Kd, out0=out, splitk=S, rownorm=(ssq, Kd, eps, rstd))
    close(out, acc * rs, 1e-2, 1e-3, "bf16 store, row norm")
    close(rstd, rs[:, 0], 1e-5, 0, "rstd")
    der, act = nan(M, N), nan(M, N)
    K.gemm(0, 0, K.EPI_BIAS_GELU, x, w, M, N, Kd, out0=der, out1=act, bias=bias, splitk=S)
    pre = (acc + bias.double()).requires_grad_(True)
    F.gelu(pre).sum().backward()
    close(act, F.gelu(pre.detach()), 1e-2, 1e-3, "gelu")
    close(der, pre.grad, 1e-2, 2e-3, "gelu'")
    res, nw = rn(M, N), rn(N)
    y, xw, sq = nan(M, N, dtype=f32), nan(M, N), nan(M, -(-N // 128), dtype=f32)
    K.gemm(0, 0, K.EPI_RESID_F32, x, w, M, N, Kd, out0=y, aux=res, bias=bias, splitk=S, next_norm=(nw, xw, sq))
    want = acc + bias.double() + res.double()
    close(y, want, 1e-5, 1e-4, "residual")
    close(xw, want * nw.double(), 1e-2, 1e-3, "next norm's operand")
    close(sq.sum(1), want.pow(2).sum(1), 1e-3, 1e-3, "sum of squares")
    # dgrad layout with saved gelu', row scale and column sums
    wt, aux, scale = w.t().contiguous(), rn(M, N).bfloat16(), torch.rand(M, device=DEV, generator=g) + 0.5
    da, col = nan(M, N), torch.ones(N, device=DEV)
    K.gemm(0, 1, K.EPI_GELU_BWD, x, wt, M, N, Kd, out0=da, aux=aux, colsum=col, rowscale=scale, splitk=S)
    want = acc * aux.double()
    close(da, want * scale.double()[:, None], 1e-2, 1e-3, "gelu' dgrad")
    close(col - 1, want.sum(0), 1e-3, 1e-3 * M ** 0.5, "column sums")
    # wgrad layout, accumulating
    dw = rn(M, N)
    before = dw.clone()
    K.gemm(1, 1, K.EPI_RED_F32, x.t().contiguous() if M % 8 == 0 else F.pad(x.t(), (0, -M % 8)).contiguous(),
           wt if N % 8 == 0 else F.pad(wt, (0, -N % 8)).contiguous(), M, N, Kd, out0=dw, splitk=S)
    close(dw, before.double() + acc, 1e-4, 1e-4 + tol, "accumulated wgrad")


@pytest.mark.parametrize("S", [1, 2, 4])
@pytest.mark.parametrize("M,V,Kd", [(1, 256, 64), (129, 200, 320), (300, 256, 1024)])
def test_split_cross_entropy(S, M, V, Kd):
    g = torch.Generator(device=DEV).manual_seed(M + S)
    x, w = (torch.randn(n, Kd, device=DEV, generator=g).bfloat16() for n in (M, V))
    labels = torch.randint(0, V, (M,), device=DEV, generator=g, dtype=torch.uint8)
    scale = torch.rand(M, device=DEV, generator=g) * 0.05 + 0.02
    loss, dl = torch.full((M,), float("nan"), device=DEV), torch.full((M, V), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.gemm(0, 0, K.EPI_CE, x, w, M, V, Kd, out0=dl, out1=loss, aux=labels, ldo=V, alpha=0.5, splitk=S, rowscale=scale)
    logits = (x.double() @ w.double().t() * scale.double()[:, None]).requires_grad_(True)
    want = F.cross_entropy(logits, labels.long(), reduction="none")
    want.sum().backward()
    close(loss, want.detach(), 1e-4, 1e-3, "loss")                      # __expf / __logf: 2^-21 of sums of 256 terms
    close(dl, logits.grad * 0.5 * scale.double()[:, None], 1e-2, 1e-4, "d logits")

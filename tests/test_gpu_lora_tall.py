"""The narrow LoRA products (csrc/lora_tall.cu): row and reduction remainders, segments, slices over a cluster."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


@pytest.mark.parametrize("M", [1, 127, 128, 129, 1537])
@pytest.mark.parametrize("K,segs,r", [(64, (64,), 8), (200, (64, 128), 16), (1024, (2048, 1024, 1024), 16), (3072, (1024,), 64), (520, (64, 64, 64, 192), 16)])
@pytest.mark.parametrize("splits", [0, 1, 2, 8])
def test_lora_tall(M, K, segs, r, splits):
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(M + K + r)
    N, nr = sum(segs), r * len(segs)
    x, dy, a, b = (torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16) for s in ((M, K), (M, N + 8), (nr, K), (N, r)))
    dy = dy[:, :N]                                        # strided rows
    st = nat._p(nat.status_word(x.device))
    out = torch.full((2, M, 72), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert nat.lib().pm_lora_tall(nat._p(x), nat.c_ll(K), nat._p(a), nat.c_ll(K), nat.c_int(0), nat.c_int(nr), nat._p(out[0]), nat.c_ll(72),
                                  nat.c_int(M), nat.c_int(K), None, nat.c_float(0.5), nat.c_int(splits), st, nat._stream()) == 0
    assert nat.lib().pm_lora_tall(nat._p(dy), nat.c_ll(N + 8), nat._p(b), nat.c_ll(r), nat.c_int(1), nat.c_int(r), nat._p(out[1]), nat.c_ll(72),
                                  nat.c_int(M), nat.c_int(N), nat._seg_ends(segs), nat.c_float(0.5), nat.c_int(splits), st, nat._stream()) == 0
    assert _rel(out[0, :, :nr], 0.5 * (x.float() @ a.float().t())) < 3e-3             # one bf16 rounding of the result
    at = 0
    for i, n in enumerate(segs):
        assert _rel(out[1, :, i * r:(i + 1) * r], 0.5 * (dy[:, at:at + n].float() @ b[at:at + n].float())) < 3e-3
        at += n
    assert (out[:, :, nr:64] == 0).all() and torch.isnan(out[:, :, 64:]).all()
    if splits == 0:
        assert _rel(nat.lora_t(x, a, 0.5)[:, :nr], out[0, :, :nr]) == 0 and _rel(nat.lora_dt(dy, b, segs, r, 0.5)[:, :nr], out[1, :, :nr]) == 0
    nat.check_status()


def test_other_ranks_keep_the_general_path():
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(1)
    for r, segs in ((32, (128, 64, 64)), (4, (128,)), (16, (40, 88))):
        N = sum(segs)
        dy = torch.randn(130, N, device="cuda", generator=g).to(torch.bfloat16)
        b = torch.randn(N, r, device="cuda", generator=g).to(torch.bfloat16)
        got, at = nat.lora_dt(dy, b, segs, r, 2.0), 0
        for i, n in enumerate(segs):
            assert _rel(got[:, i * r:(i + 1) * r], 2 * dy[:, at:at + n].float() @ b[at:at + n].float()) < 3e-3, (r, i)
            at += n


@pytest.mark.parametrize("M", [100, 129, 300, 1537])
@pytest.mark.parametrize("segs,r,K", [((256, 128, 128), 16, 256), ((192,), 16, 136), ((64, 64), 32, 520), ((64, 128), 16, 64)])
@pytest.mark.parametrize("transposed", [True, False])
def test_lora_layer_in_one_call(M, segs, r, K, transposed):
    """Forward and gradients of a layer through the one-call entries and, outside of their rules, through the single products."""
    from pmetal_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(M + K + r)
    N, nr = sum(segs), r * len(segs)
    f = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, res, dy = f(M, K).to(torch.bfloat16).requires_grad_(True), f(M, N).to(torch.bfloat16), f(M, N).to(torch.bfloat16)
    w = (f(N, K) * K ** -0.5).to(torch.bfloat16)
    a, b = (f(nr, K) * K ** -0.5).requires_grad_(True), (f(N, r) * 0.1).requires_grad_(True)
    y = ops.lora_linear(x, w, w.t().contiguous() if transposed else None, a, b, segs, r, 2.0, res)
    got = torch.autograd.grad(y, (x, a, b), dy)
    xr, ar, br = (t.detach().to(torch.bfloat16).float().requires_grad_(True) for t in (x, a, b))
    parts, at = [], 0
    for i, n in enumerate(segs):
        parts.append(2.0 * (xr @ ar[i * r:(i + 1) * r].t()) @ br[at:at + n].t())
        at += n
    want = xr @ w.float().t() + res.float() + torch.cat(parts, -1)
    assert _rel(y.detach(), want.detach()) < 4e-3                    # bf16 t and y
    for p, q in zip(got, torch.autograd.grad(want, (xr, ar, br), dy.float())):
        assert _rel(p, q) < 6e-3                                     # bf16 dt, t and dx


# ranks whose segments are wider than one tile of the general path, together or each; padding columns beside a multiple of 8
@pytest.mark.parametrize("segs,r", [((128, 64), 64), ((256, 128, 128), 64), ((256,), 128), ((128, 128), 96), ((128, 64, 64), 24), ((96, 32), 64),
                                    ((192,), 72)])
@pytest.mark.parametrize("M", [100, 300])
def test_gradients_of_wide_ranks(segs, r, M):
    from pmetal_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(M + r)
    K, N, nr = 136, sum(segs), r * len(segs)
    f = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, dy = f(M, K).to(torch.bfloat16).requires_grad_(True), f(M, N).to(torch.bfloat16)
    w = (f(N, K) * K ** -0.5).to(torch.bfloat16)
    a, b = (f(nr, K) * K ** -0.5).requires_grad_(True), (f(N, r) * 0.1).requires_grad_(True)
    y = ops.lora_linear(x, w, None, a, b, segs, r, 2.0)
    poison = [torch.full((n,), float("nan"), dtype=torch.bfloat16, device="cuda") for n in (M * 64, M * 128, M * 192, M * 256) for _ in range(8)]
    del poison                                             # what the products allocate next holds NaN where they do not write
    got = torch.autograd.grad(y, (x, a, b), dy)
    xr, ar, br = (t.detach().to(torch.bfloat16).float().requires_grad_(True) for t in (x, a, b))
    parts, at = [], 0
    for i, n in enumerate(segs):
        parts.append(2.0 * (xr @ ar[i * r:(i + 1) * r].t()) @ br[at:at + n].t())
        at += n
    want = xr @ w.float().t() + torch.cat(parts, -1)
    assert _rel(y.detach(), want.detach()) < 4e-3                    # bf16 t and y
    for name, p, q in zip(("x", "a", "b"), got, torch.autograd.grad(want, (xr, ar, br), dy.float())):
        assert _rel(p, q) < 6e-3, name                               # bf16 dt, t and dx

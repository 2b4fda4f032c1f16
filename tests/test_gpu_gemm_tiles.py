"""The CTA-pair GEMM at the edges of its tiles, of its staged epilogue and of its tile order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _near(y, ref, what):
    """bf16 rounds to 2^-9 of a value; the fp32 sums of up to 9728 products of unit size in all stay within 1e-3."""
    err = (y.float() - ref).abs()
    assert bool((err <= ref.abs() * 2.0 ** -8 + 1e-3).all()), f"{what}: {float(err.max())}"


# last row block of 1 .. 255 rows, columns that end inside a 64-wide piece, one and many groups of 16 row blocks (the last
# one short), one k block and many, both tile widths, LoRA segments that end on multiples of 128 but not of 256
@pytest.mark.parametrize("M,N,K,segs", [(256, 256, 64, ()), (257, 264, 72, ()), (511, 1000, 1024, ()), (4865, 1024, 136, ()),
                                        (2048, 1024, 2048, (1024,)), (1300, 640, 320, (256, 128, 256)), (8193, 512, 200, (256, 256)),
                                        (300, 4096, 9728, (2048, 1024, 1024))])
def test_pair_gemm_tile_edges(M, N, K, segs):
    from pmetal_b200.ops import native as nat
    torch.manual_seed(M + N)
    x, w, res = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(M, N)
    ref = x.float() @ w.float().t()
    _near(nat.gemm(x, w), ref, "plain")
    # the residual lives in a wider matrix, the result goes into one: neither may be written beside its columns
    wide, out = _rand(M, N + 64), torch.full((M, N + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    nat.gemm(x, w, alpha=0.5, residual=wide[:, 8:N + 8], out=out[:, 16:N + 16])
    _near(out[:, 16:N + 16], 0.5 * ref + wide[:, 8:N + 8].float(), "strided residual and result")
    assert bool((out[:, :16] == 7).all()) and bool((out[:, N + 16:] == 7).all())
    same = res.clone()
    nat.gemm(x, w, residual=same, out=same)
    _near(same, ref + res.float(), "residual in place")
    if segs:
        a, b = _rand(16 * len(segs), K, scale=K ** -0.5), _rand(N, 16, scale=0.2)
        t = nat.lora_t(x, a, 2.0)
        want, at = ref + res.float(), 0
        for i, n in enumerate(segs):
            want[:, at:at + n] += t[:, 16 * i:16 * i + 16].float() @ b[at:at + n].float().t()
            at += n
        _near(nat.gemm_lora(x, w, t, b, segs, 16, res), want, "segments")
    nat.check_status()


# tiles that lie past the stored columns altogether, several to a pair (one pair walks all of them), either tile width
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("M,N,K,stored", [(512, 1024, 128, 64), (300, 640, 192, 8), (768, 1536, 64, 520),
                                            (512, 1024, 128, 100), (768, 1536, 64, 513)])
def test_pair_gemm_stores_fewer_columns_than_it_computes(M, N, K, stored, residual):
    from pmetal_b200.ops import native as nat
    torch.manual_seed(N)
    x, w, res = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(M, N)
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    nat.raw_gemm(x, 0, K, M, w, 0, K, N, out, 0, N, M, N, K, R=res if residual else None, ldr=N if residual else 0, n_store=stored, bn=256,
                 max_ctas=2)
    ref = x.float() @ w.float().t()
    _near(out[:, :stored], (ref + res.float() if residual else ref)[:, :stored], "stored columns")
    assert bool((out[:, stored:] == 7).all())
    nat.check_status()


@pytest.mark.parametrize("N", [500, 251, 1023])
def test_pair_gemm_into_a_wider_matrix(N):
    """The last columns of the result end inside 16 bytes: what lies beside them in the same row stays."""
    from pmetal_b200.ops import native as nat
    torch.manual_seed(N)
    x, w, wide = _rand(520, 256), _rand(N, 256, scale=1 / 16), _rand(520, 1032)
    out = torch.full((520, 1032), 7.0, dtype=torch.bfloat16, device="cuda")
    nat.gemm(x, w, residual=wide[:, :N], out=out[:, :N])
    _near(out[:, :N], x.float() @ w.float().t() + wide[:, :N].float(), "result")
    assert bool((out[:, N:] == 7).all())
    nat.check_status()


def test_the_pair_kernel_can_be_switched_off(monkeypatch):
    """Without it neither a LoRA layer nor a prompt launches it, and the results stay."""
    from pmetal_b200.models.config import ModelArgs
    from pmetal_b200.models.decoder import DecoderLM
    from pmetal_b200.models.generation import Generator
    from pmetal_b200.ops import functional as ops
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(2)
    f = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, w, a, b = f(300, 256).bfloat16().requires_grad_(True), f(256, 256).bfloat16() / 16, f(16, 256) / 16, f(256, 16) / 4
    a.requires_grad_(True), b.requires_grad_(True)
    m = DecoderLM(ModelArgs(vocab_size=64, hidden_size=256, intermediate_size=256, num_hidden_layers=2, num_attention_heads=2,
                            num_key_value_heads=1, head_dim=128)).init_weights(0.05, 1).to("cuda").to(torch.bfloat16).eval()
    for p in m.parameters():
        p.requires_grad_(False)

    class Counting:
        def __init__(self, real):
            self.real, self.names = real, []

        def __getattr__(self, name):
            self.names.append(name)
            return getattr(self.real, name)

    def both():
        counter = Counting(nat.lib())
        with monkeypatch.context() as mp:
            mp.setattr(nat, "lib", lambda: counter)
            mp.setattr(nat, "_LORA_ARGS", {})
            y = ops.lora_linear(x, w, None, a, b, (256,), 16, 1.0)
            grads = torch.autograd.grad(y.float().square().sum(), (x, a, b))
            gen = Generator(m, num_blocks=16, cuda_graphs=False)
            out = [y, *grads, gen.prefill([gen.new_seq()], [list(range(60)) * 5])]
        return [t.detach().float() for t in out], set(counter.names)
    on, names = both()
    assert names & {"pm_lora_linear_fwd", "pm_lora_linear_bwd", "pm_layer_stack"} == {"pm_lora_linear_fwd", "pm_lora_linear_bwd", "pm_layer_stack"}
    monkeypatch.setattr(nat, "USE_2SM", False)
    off, names = both()
    assert not names & {"pm_lora_linear_fwd", "pm_lora_linear_bwd", "pm_layer_stack", "pm_gemm_bf16_2sm"}
    for p, q in zip(on, off):
        assert float((p - q).norm() / q.norm()) < 2e-2               # two layers of bf16 activations
    nat.check_status()

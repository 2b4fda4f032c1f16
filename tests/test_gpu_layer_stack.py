"""Few-row linear layers (csrc/gemm_skinny.cu) and the one-call layer stack (csrc/layer_stack.cu)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


# rows beside the tile widths 16, 32, 64, 128; columns that end inside a tile; K that ends inside a k block or inside a split
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 1032), (72, 520), (1024, 3072)])
@pytest.mark.parametrize("splits", [0, 1, 2, 8])
@pytest.mark.parametrize("swiglu", [0, 1])
def test_skinny_linear(M, N, K, splits, swiglu):
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn((1 + swiglu) * N, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    res = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    y = torch.full((M, N + 8), float("nan"), dtype=torch.bfloat16, device="cuda")
    rc = nat.lib().pm_linear_skinny(nat._p(x), nat.c_ll(K), nat._p(w), nat.c_ll(K), nat._p(y), nat.c_ll(N + 8), nat._p(res), nat.c_ll(N),
                                    nat.c_int(M), nat.c_int(N), nat.c_int(K), nat.c_int(swiglu), nat.c_float(0.5), nat.c_int(splits),
                                    nat.c_int(0), nat._p(nat.status_word(x.device)), nat._stream())
    assert rc == 0
    want = 0.5 * (x.float() @ w.float().t())
    if swiglu:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    want = want + res.float()
    assert _rel(y[:, :N], want) < 3e-3            # one bf16 rounding of the result
    assert torch.isnan(y[:, N:]).all()
    nat.check_status()


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("qk_norm", [True, False])
@pytest.mark.parametrize("lens", [[1], [3, 16], [90, 39], [129], [257, 70, 64]])
def test_layer_stack_matches_the_layer_by_layer_forward(quant, qk_norm, lens, monkeypatch):
    """Prompts and decode steps through one call of the runtime against the same model in fp32 PyTorch."""
    from pmetal_b200.models.config import ModelArgs
    from pmetal_b200.models.decoder import DecoderLM
    from pmetal_b200.models.generation import Generator
    from pmetal_b200.ops import native as nat
    cfg = ModelArgs(vocab_size=512, hidden_size=256, intermediate_size=520, num_hidden_layers=2, num_attention_heads=4,
                    num_key_value_heads=2, head_dim=128, qk_norm=qk_norm)
    m = DecoderLM(cfg).init_weights(0.05, 5).to("cuda").to(torch.bfloat16).eval()
    for p in m.parameters():
        p.requires_grad_(False)
    calls = []
    monkeypatch.setattr(nat, "layer_stack", lambda *a, _f=nat.layer_stack: calls.append(1) or _f(*a))
    g = torch.Generator().manual_seed(3)
    prompts = [torch.randint(0, 512, (n + 2,), generator=g).tolist() for n in lens]
    gen = Generator(m, cache=m.new_cache(32, quant=quant), cuda_graphs=False)
    seqs = [gen.new_seq() for _ in lens]
    got = [gen.prefill(seqs, [p[:-2] for p in prompts])]
    for k in (2, 1):
        got.append(gen.decode_step(seqs, torch.tensor([p[-k] for p in prompts], device="cuda")))
    assert len(calls) == 3
    ref = DecoderLM(cfg).init_weights(0.05, 5).to(torch.bfloat16).float().eval()
    for i, p in enumerate(prompts):
        with torch.no_grad():
            want = ref(torch.tensor([p]))[0]
        for k in range(3):
            # two layers of bf16 activations (about six roundings of 2^-9 each); the int8 cache adds 1/254 of a group's maximum
            assert _rel(got[k][i].cpu(), want[len(p) - 3 + k]) < (3e-2 if quant else 2e-2), (i, k)
    nat.check_status()


def test_layer_stack_leaves_other_models_alone():
    from pmetal_b200.core.config import LoraConfig
    from pmetal_b200.lora import apply_lora
    from pmetal_b200.models.config import ModelArgs
    from pmetal_b200.models.decoder import DecoderLM
    def make(**kw):
        cfg = ModelArgs(vocab_size=64, hidden_size=128, intermediate_size=128, num_hidden_layers=1, num_attention_heads=2,
                        num_key_value_heads=1, head_dim=128, **kw)
        m = DecoderLM(cfg, torch.bfloat16, "cuda")
        for p in m.parameters():
            p.requires_grad_(False)
        return m
    m = make()
    assert m._stack_addresses(m.new_cache(4)) is not None and m._stack_addresses(m.new_cache(4, quant="int8")) is not None
    assert m._stack_addresses(m.new_cache(4, quant="tq4")) is None and m._stack_addresses(m.new_cache(4, window=64)) is None
    assert make(attention_bias=True)._stack_addresses(m.new_cache(4)) is None
    m.layers[0].mlp.down_proj.weight.requires_grad_(True)
    assert m._stack_addresses(m.new_cache(4)) is None
    m = make()
    apply_lora(m, LoraConfig(r=8, alpha=8, target_modules=["q_proj"]), seed=0)
    assert m._stack_addresses(m.new_cache(4)) is None


@pytest.mark.parametrize("M,N", [(16, 4096), (64, 24), (65, 4096), (65, 1024), (128, 136)])
def test_gemm_on_few_rows_takes_either_kernel(M, N):
    """Strided operands and results, with and without a residual, on both sides of the rule that picks the few-row kernel."""
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, 776, device="cuda", generator=g).to(torch.bfloat16)[:, :768]
    w = (torch.randn(N, 768, device="cuda", generator=g) * 768 ** -0.5).to(torch.bfloat16)
    res = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    want = x.float() @ w.float().t()
    assert _rel(nat.gemm(x, w), want) < 3e-3 and _rel(nat.gemm(x, w, residual=res), want + res.float()) < 3e-3
    assert _rel(nat.gemm_lora(x, w, None, None, (N,), 0, res), want + res.float()) < 3e-3
    h = torch.randn(3, 768, device="cuda", generator=g).to(torch.bfloat16)
    nw = torch.rand(768, device="cuda", generator=g).to(torch.bfloat16)
    normed = h.float() * torch.rsqrt(h.float().square().mean(-1, keepdim=True) + 1e-6) * nw.float()
    assert _rel(nat.few_row_head(h, w, nw, 1e-6), normed @ w.float().t()) < 5e-3
    nat.check_status()

"""Tile edges of the tcgen05 attention kernels: the packed forward / backward and the paged forward against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.detach().float() - b.detach().float()).norm() / b.detach().float().norm())


def _dense(q, k, v, first, limit, scale):
    """fp32 attention of q [T, hq, d]: query i sees the keys first[i] .. limit[i]."""
    rep = q.shape[1] // k.shape[1]
    kk, vv = (t.float().repeat_interleave(rep, 1).transpose(0, 1) for t in (k, v))
    s = q.float().transpose(0, 1) @ kk.transpose(1, 2) * scale
    j = torch.arange(k.shape[0], device=q.device)[None]
    s = s.masked_fill(~((j >= first[:, None]) & (j <= limit[:, None])), float("-inf"))
    return (s.softmax(-1) @ vv).transpose(0, 1)


# (kv lengths, new tokens): one token beside a prompt, ends on and beside the 64-token block and the 128-row tile, an odd number of blocks
PAGED = [([1, 130], [1, 130]), ([64, 65, 63], [64, 65, 63]), ([129, 700, 256], [128, 1, 200]), ([1000], [333]), ([127, 128, 129, 193], [100, 128, 129, 65])]


@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 4), (16, 4), (8, 1)])
@pytest.mark.parametrize("lens,qlens", PAGED)
def test_paged_prompt_attention(hq, hkv, lens, qlens):
    from pmetal_b200.models.kv_cache import PagedKVCache
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + hq)
    cache = PagedKVCache(1, hkv, 128, 48)
    cache.free = [b for b in torch.randperm(48, generator=torch.Generator().manual_seed(3)).tolist()]
    for t in (cache.k[0], cache.v[0]):
        t.copy_(torch.randn(t.shape, device="cuda", generator=g))
    for i, (n, m) in enumerate(zip(lens, qlens)):
        cache.add_sequence(i)
        if n > m:
            cache.reserve(i, n - m)
    meta = cache.prepare(list(range(len(lens))), qlens)
    q = torch.randn(sum(qlens), hq, 128, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    rc = nat.lib().pm_paged_attn_tc(nat._p(q), nat._p(cache.k[0]), nat._p(cache.v[0]), nat._p(out), nat._p(meta.block_table),
                                    nat._p(meta.seq_lens), nat._p(meta.q_start), nat._p(meta.q_lens), nat.c_int(len(lens)),
                                    nat.c_int(meta.block_table.shape[1]), nat.c_int(48), nat.c_int(sum(qlens)), nat.c_int(max(qlens)),
                                    nat.c_int(hq), nat.c_int(hkv), nat.c_float(128 ** -0.5), nat._p(nat.status_word(q.device)), nat._stream())
    assert rc == 0
    at = 0
    for i, (n, m) in enumerate(zip(lens, qlens)):
        k, v = cache.gather(0, i)
        lim = torch.arange(n - m, n, device="cuda")
        want = _dense(q[at:at + m], k, v, torch.zeros_like(lim), lim, 128 ** -0.5)
        # bf16 probabilities and outputs: 2^-9 each, relative to the row
        assert _rel(out[at:at + m], want) < 6e-3, (i, n, m)
        at += m
    nat.check_status()


def _paged_decode(q, cache, meta, splits=0):
    from pmetal_b200.ops import native as nat
    p, c = nat._p, nat.c_int
    out = torch.full_like(q, float("nan"))
    scales = (cache.k_scale[0], cache.v_scale[0]) if cache.quant else (None, None)
    rc = nat.lib().pm_paged_decode(p(q), p(cache.k[0]), p(cache.v[0]), p(scales[0]), p(scales[1]), p(out), p(meta.block_table),
                                   p(meta.seq_lens), p(meta.q_start), p(meta.q_lens), c(meta.block_table.shape[0]),
                                   c(meta.block_table.shape[1]), c(cache.num_blocks), c(meta.max_q), c(q.shape[1]), c(cache.hkv),
                                   nat.c_float(128 ** -0.5), c(splits), p(nat.status_word(q.device)), nat._stream())
    assert rc == 0
    return out


# (kv lengths, new tokens): ends on and beside the 16-key quarters and the 64-key blocks, fewer blocks than slices, several tokens
DECODE = [([1, 15, 16, 17], [1, 1, 1, 1]), ([63, 64, 65, 700], [1, 1, 1, 1]), ([130, 5], [5, 2]), ([2100], [8])]


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("hq,hkv", [(2, 2), (4, 2), (8, 1), (6, 2)])
@pytest.mark.parametrize("lens,qlens", DECODE)
@pytest.mark.parametrize("splits", [0, 1, 2, 8])
def test_paged_decode_attention(quant, hq, hkv, lens, qlens, splits):
    from pmetal_b200.models.kv_cache import PagedKVCache
    from pmetal_b200.ops import native as nat
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + hq)
    cache = PagedKVCache(1, hkv, 128, 64, quant=quant)
    cache.free = torch.randperm(64, generator=torch.Generator().manual_seed(3)).tolist()
    for i, (n, m) in enumerate(zip(lens, qlens)):
        cache.add_sequence(i)
        if n > m:
            cache.reserve(i, n - m)
    meta = cache.prepare(list(range(len(lens))), qlens)
    every = torch.arange(64 * 64, device="cuda")
    k, v = (torch.randn(64 * 64, hkv, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    cache.write_reference(0, k, v * 0.01, every)         # small values: the scales of the int8 cache matter
    q = torch.randn(sum(qlens), hq, 128, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    p = nat._p
    scales = (cache.k_scale[0], cache.v_scale[0]) if quant else (None, None)
    rc = nat.lib().pm_paged_decode(p(q), p(cache.k[0]), p(cache.v[0]), p(scales[0]), p(scales[1]), p(out), p(meta.block_table),
                                   p(meta.seq_lens), p(meta.q_start), p(meta.q_lens), nat.c_int(len(lens)),
                                   nat.c_int(meta.block_table.shape[1]), nat.c_int(64), nat.c_int(max(qlens)), nat.c_int(hq),
                                   nat.c_int(hkv), nat.c_float(128 ** -0.5), nat.c_int(splits), p(nat.status_word(q.device)), nat._stream())
    assert rc == 0
    cache.compute_dtype = torch.float32                  # the oracle reads codes times scales unrounded
    at = 0
    for i, (n, m) in enumerate(zip(lens, qlens)):
        kk, vv = cache.gather(0, i)
        lim = torch.arange(n - m, n, device="cuda")
        want = _dense(q[at:at + m], kk, vv, torch.zeros_like(lim), lim, 128 ** -0.5)
        assert _rel(out[at:at + m], want) < 5e-3, (i, n, m)      # bf16 probabilities and outputs: 2^-9 each
        at += m


@pytest.mark.parametrize("hq,hkv", [(2, 2), (4, 2), (8, 1)])
@pytest.mark.parametrize("n,splits", [(64, 1), (333, 2), (2100, 8)])
def test_paged_decode_keeps_its_probabilities(hq, hkv, n, splits):
    """Values of opposite sign at keys that nearly agree: what is left of the sum is about 2 % of a probability, where a probability
    rounded to bf16 (2^-9) would leave errors of several per cent of it."""
    from pmetal_b200.models.kv_cache import PagedKVCache
    g = torch.Generator(device="cuda").manual_seed(n + hq)
    cache = PagedKVCache(1, hkv, 128, 48)
    cache.add_sequence(0)
    if n > 1:
        cache.reserve(0, n - 1)
    meta = cache.prepare([0], [1])
    k, v = (torch.randn(48 * 64, hkv, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    k[1::2] = (k[::2].float() + 0.02 * torch.randn(k[::2].shape, device="cuda", generator=g)).to(torch.bfloat16)
    v[1::2] = -v[::2]
    cache.write_reference(0, k, v, torch.arange(48 * 64, device="cuda"))
    q = torch.randn(1, hq, 128, device="cuda", generator=g).to(torch.bfloat16)
    out = _paged_decode(q, cache, meta, splits)
    kk, vv = (t.double().repeat_interleave(hq // hkv, 1) for t in cache.gather(0, 0))
    s = torch.einsum("hd,jhd->hj", q[0].double(), kk) * 128 ** -0.5
    want = torch.einsum("hj,jhd->hd", s.softmax(-1), vv)
    assert float((out[0].double() - want).norm() / want.norm()) < 4e-3       # one bf16 rounding of the output


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("left", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("lens,qlens", [([1, 15, 33, 64, 190], [1, 1, 1, 1, 1]), ([70, 9], [5, 8])])
def test_paged_decode_ignores_what_lies_past_the_keys(quant, left, lens, qlens):
    """A block that another sequence has given back keeps its contents: they do not reach the sequence that has it now."""
    from pmetal_b200.models.kv_cache import PagedKVCache
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    cache = PagedKVCache(1, 2, 128, 16, quant=quant)
    for i, (n, m) in enumerate(zip(lens, qlens)):
        cache.add_sequence(i)
        if n > m:
            cache.reserve(i, n - m)
    meta = cache.prepare(list(range(len(lens))), qlens)
    every = torch.arange(16 * 64, device="cuda")
    k, v = (torch.randn(16 * 64, 2, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    cache.write_reference(0, k, v, every)
    q = torch.randn(sum(qlens), 4, 128, device="cuda", generator=g).to(torch.bfloat16)
    clean = _paged_decode(q, cache, meta)
    held = torch.cat([torch.tensor(cache.seqs[i].blocks)[torch.arange(n) // 64] * 64 + torch.arange(n) % 64 for i, n in enumerate(lens)])
    other = torch.ones(16 * 64, dtype=torch.bool)
    other[held] = False
    for t in ((cache.k_scale[0], cache.v_scale[0]) if quant else (cache.k[0], cache.v[0])):
        t.view(16 * 64, -1)[other.cuda()] = left
    got = _paged_decode(q, cache, meta)
    assert bool(torch.isfinite(clean).all()) and bool((got == clean).all())


def test_paged_dispatch_keeps_small_steps_on_the_split_kernel():
    from pmetal_b200.ops.native import _paged_on_tensor_cores as tc
    assert tc(1, 2048, 2048, 16, 8) and tc(6, 700, 700, 16, 8) and tc(1, 512, 12000, 16, 8)
    assert not tc(64, 1, 8000, 16, 8) and not tc(1, 37, 37, 16, 8) and not tc(1, 128, 12000, 16, 8) and not tc(1, 2048, 2048, 12, 4)


@pytest.mark.parametrize("lens", [[1, 127, 1, 128, 200], [300], [129, 64, 1, 1, 400, 55], [513]])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 2)])
def test_packed_attention_at_tile_edges(lens, hq, hkv):
    from pmetal_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    T = sum(lens)
    q, k, v = (torch.randn(T, h, 128, device="cuda", generator=g).to(torch.bfloat16).requires_grad_(True) for h in (hq, hkv, hkv))
    start = torch.repeat_interleave(torch.tensor([sum(lens[:i]) for i in range(len(lens))]), torch.tensor(lens)).int().cuda()
    w = torch.randn(T, hq, 128, device="cuda", generator=g)
    o = ops._AttnCoreFn.apply(q, k, v, start, 128 ** -0.5, 0)
    grads = torch.autograd.grad((o.float() * w).sum(), (q, k, v))
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    want = _dense(qf, kf, vf, start.long(), torch.arange(T, device="cuda"), 128 ** -0.5)
    ref = torch.autograd.grad((want * w.to(torch.bfloat16).float()).sum(), (qf, kf, vf))
    assert _rel(o, want) < 6e-3
    # bf16 P, dS, O and dO enter the products: a handful of 2^-9 roundings
    for a, b in zip(grads, ref):
        assert _rel(a, b) < 1.5e-2

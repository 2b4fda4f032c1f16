"""Sampling of rows that are cut over a cluster: slice edges, ties, masked logits and thresholds against PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# vocabularies that give 1, 2, 4 and 8 slices, ends inside a group of eight, rows off 16-byte boundaries
@pytest.mark.parametrize("V", [37, 8192, 16391, 50257, 65541, 151936])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B", [1, 5, 80])
def test_greedy_rows(V, dtype, B):
    from pmetal_b200.models.sampling import Sampler, SamplingParams
    g = torch.Generator(device="cuda").manual_seed(V + B)
    x = torch.randn(B, V, device="cuda", generator=g).to(dtype)
    x[0, V // 2] = x[0, V - 1] = 9.0                      # a tie over slices: the smaller index
    if B > 1:
        x[1] = float("-inf")
        x[1, V - 1] = -3.0                                # everything else masked
        x[2, : V // 2] = float("-inf")
    ids, lp = Sampler(SamplingParams.greedy(), "cuda").sample(x, return_logprobs=True)
    assert int(ids[0]) == V // 2 and torch.equal(x.gather(1, ids[:, None])[:, 0], x.max(-1).values)
    want = torch.log_softmax(x.double(), -1).gather(1, ids[:, None])[:, 0]
    assert float((lp.double() - want).abs().max()) < 1e-4          # fp32 sums of 150k terms and __expf


@pytest.mark.parametrize("V", [300, 16391, 151936])
@pytest.mark.parametrize("kw", [dict(top_k=20, top_p=1.0), dict(top_k=0, top_p=0.4), dict(top_k=50, top_p=0.7), dict(top_k=0, top_p=1.0, min_p=0.2)])
def test_drawn_tokens_survive_the_filters(V, kw):
    from pmetal_b200.models.sampling import Sampler, SamplingParams, filtered_logprobs
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(6, V, device="cuda", generator=g) * 3).to(torch.bfloat16)
    p = SamplingParams(temperature=0.8, do_sample=True, seed=5, **{"min_p": 0.0, **kw})
    s = Sampler(p, "cuda")
    keep = filtered_logprobs(x.float(), p)
    for _ in range(8):
        ids, lp = s.sample(x, return_logprobs=True)
        floor = keep.masked_fill(keep == float("-inf"), 1e9).amin(-1)
        at = torch.log_softmax(x.float(), -1).gather(1, ids[:, None])[:, 0]
        assert bool((at >= floor - 0.07).all())            # bf16 logits tie at the edge of a nucleus; one step there is 2^-4
        q = torch.log_softmax(keep / 0.8, -1).gather(1, ids[:, None])[:, 0]
        ok = q > float("-inf")
        assert float((lp - q)[ok].abs().max()) < 0.05      # a tied token more or less in the nucleus


@pytest.mark.parametrize("V", [37, 16391, 151936])
@pytest.mark.parametrize("kw", [dict(temperature=0.0), dict(temperature=0.8, do_sample=True, top_k=5), dict(temperature=1.0, do_sample=True, top_p=0.5)])
@pytest.mark.parametrize("bad", [float("-inf"), float("nan")])
def test_rows_without_a_choice(V, kw, bad):
    """A row in which every logit is -inf or NaN gives a token of the vocabulary; its neighbours are what they are alone."""
    from pmetal_b200.models.sampling import Sampler, SamplingParams
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(3, V, device="cuda", generator=g)
    x[1] = bad
    x[2, 1:] = float("-inf")
    ids, lp = Sampler(SamplingParams(seed=3, **kw), "cuda").sample(x, return_logprobs=True)
    assert int(ids[1]) == 0 and bool(torch.isnan(lp[1])) and int(ids[2]) == 0 and abs(float(lp[2])) < 1e-5
    assert 0 <= int(ids[0]) < V and bool(torch.isfinite(lp[0]))

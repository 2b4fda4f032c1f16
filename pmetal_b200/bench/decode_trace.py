"""Tiny decode runs for profiling.

    python -m pmetal_b200.bench.decode_trace [--tokens 6]             one sequence, a few greedy tokens, no CUDA graphs
                                                                       (launch lists under a profiler)
    python -m pmetal_b200.bench.decode_trace --phases [--batch 1]     device time of every kernel of a decode step, as the
                                                                       profiler's activity records give it
"""
import argparse
import json
import os


def phase_trace(model, batch: int, prompt_len: int = 128) -> dict:
    """Median duration (us) and launches per step of every kernel of a decode step, and the span of a whole step. Chained kernels
    start before their predecessor has ended, so the durations overlap."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    from ..models.generation import Generator
    gen = Generator(model, num_blocks=1024, cuda_graphs=False)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, model.cfg.vocab_size, (prompt_len,), generator=g).tolist() for _ in range(batch)]
    seqs = [gen.new_seq() for _ in prompts]
    ids = gen.prefill(seqs, prompts).argmax(-1)
    for _ in range(3):
        ids = gen.decode_step(seqs, ids).argmax(-1)
    steps = 3
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(steps):
            ids = gen.decode_step(seqs, ids).argmax(-1)
        torch.cuda.synchronize()
    times = {}
    events = [e for e in prof.events() if str(e.device_type).endswith("CUDA")]
    for e in events:
        name = e.name.split("(")[0].removeprefix("void ")
        times.setdefault(name, []).append(e.time_range.elapsed_us())
    out = {n: {"us": round(sorted(t)[len(t) // 2], 2), "per_step": round(len(t) / steps, 2)} for n, t in times.items()}
    out["step_us"] = round((max(e.time_range.end for e in events) - min(e.time_range.start for e in events)) / steps, 1)
    return out


def add_arguments(ap) -> None:
    ap.add_argument("--tokens", type=int, default=6)
    ap.add_argument("--model", default="random:qwen3-0.6b")
    ap.add_argument("--phases", action="store_true")
    ap.add_argument("--batch", type=int, default=1)


def main(argv=None, args=None) -> int:
    """Also reachable as ``pmetal bench-decode`` (which passes its parsed arguments as ``args``)."""
    os.environ.setdefault("PMETAL_DECODE_GRAPHS", "0")      # eager launches: one kernel per launch under a profiler
    import torch

    from ..models.generation import Generator
    from ..models.loader import load_pretrained
    from ..models.sampling import SamplingParams
    a = args
    if a is None:
        ap = argparse.ArgumentParser()
        add_arguments(ap)
        a = ap.parse_args(argv)
    m, _, _ = load_pretrained(a.model, dtype=torch.bfloat16, device="cuda")
    m.eval()
    for p in m.parameters():
        p.requires_grad_(False)
    if a.phases:
        print(json.dumps({"batch": a.batch, **phase_trace(m, a.batch)}))
        return 0
    g = Generator(m, num_blocks=256, cuda_graphs=False)
    r = g.generate([list(range(1, 65))], SamplingParams.greedy(a.tokens))
    torch.cuda.synchronize()
    print("generated", r.generated_tokens)
    return 0


if __name__ == "__main__":
    raise SystemExit(main())

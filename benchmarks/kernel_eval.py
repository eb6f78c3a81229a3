"""Stand-alone timing of the ranking kernels: ``python benchmarks/kernel_eval.py``.

Times the counting kernel that ``FusedRanker`` launches (``rank_count``, and with ``--band`` its form on split operands with
an undecided band, three GEMMs) and the top-k search with CUDA events after warm-up, flushing L2 between launches, and
reports the achieved tensor throughput (``2·B·|E|·D`` FLOP per GEMM) as a fraction of the cuBLAS bf16 figure in
``MEASURED_PEAKS.json``.  With ``--compare`` it also times the PyTorch formulation of the same counts (``torch.mm`` per 1024
queries + comparison + row sum).  It is the small, self-terminating program used for ``ncu`` captures of these kernels."""
from __future__ import annotations

import argparse
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))  # run from a source checkout

import torch

from dice_embeddings_b200.utils.profiling import measured_peaks
from dice_embeddings_b200.ops import kernels as K
from dice_embeddings_b200.ops.eval_rank import FusedRanker


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--queries", type=int, default=4096)
    ap.add_argument("--entities", type=int, default=262144)
    ap.add_argument("--d", type=int, default=256)
    ap.add_argument("--iters", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--topk", type=int, default=0, help="also time top-k mode with this k on the first 256 queries")
    ap.add_argument("--band", action="store_true", help="also time the counting kernel on split operands")
    ap.add_argument("--topk_queries", type=int, default=256)
    ap.add_argument("--compare", action="store_true")
    a = ap.parse_args()
    dev = torch.device("cuda:0")
    torch.manual_seed(0)
    q = (torch.randn(a.queries, a.d, device=dev) * 0.3).to(torch.bfloat16)
    y = (torch.randn(a.entities, a.d, device=dev) * 0.3).to(torch.bfloat16)
    tgt = torch.randint(0, a.entities, (a.queries,), device=dev, dtype=torch.int32)
    ts = torch.zeros(a.queries, device=dev)
    greater = torch.zeros(a.queries, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    K.eval_sparse(q, y, tgt, ts, None)
    pk = measured_peaks()

    def timed(fn, iters):
        for _ in range(a.warmup):
            fn()
        torch.cuda.synchronize()
        ms = 0.0
        for _ in range(iters):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            ms += e0.elapsed_time(e1)
        return ms / iters

    def report(name, ms, gemms):
        tf = 2.0 * gemms * a.queries * a.entities * a.d / (ms * 1e-3) / 1e12
        print(f"{name}  B={a.queries} E={a.entities} D={a.d}: {ms * 1e3:9.1f} us  {tf:7.1f} TFLOP/s  "
              f"{tf / pk['bf16_tflops']:.2f} of {pk['source']} ({pk['bf16_tflops']:.0f})")

    report("rank_count", timed(lambda: K.rank_count(q, y, ts, tgt, greater, status), a.iters), 1)
    if a.band:
        q32, y32 = q.float() + 1e-3 * torch.randn_like(q.float()), y.float() + 1e-3 * torch.randn_like(y.float())
        yh, yl, _, _ = K.split_rows(y32, a.d)
        qh, ql, _, margin = K.split_rows(q32, a.d, margin_factor=float(y32.norm(dim=1).max()) * FusedRanker.MARGIN[a.d])
        K.eval_sparse(q32, y32, tgt, ts, None)
        rows, cols = (torch.empty(1 << 24, dtype=torch.int32, device=dev) for _ in range(2))
        count = torch.zeros(1, dtype=torch.int64, device=dev)

        def banded():
            count.zero_()
            K.rank_count(qh, yh, ts, tgt, greater, status, x_lo=ql, y_lo=yl, margin=margin, band_rows=rows, band_cols=cols,
                         band_count=count)
        report("rank_count, split operands", timed(banded, a.iters), 3)
        print(f"   undecided: {int(count) / (a.queries * a.entities):.1e} of the pairs")
    if a.topk:
        r = FusedRanker(y)
        n = min(a.topk_queries, a.queries)
        ms = timed(lambda: r.topk(q[:n], a.topk), max(a.iters // 2, 1))
        r.check()
        print(f"top-{a.topk} of {n} queries over {a.entities} entities: {ms * 1e3:9.1f} us")
    if a.compare:
        def torch_counts():
            out = []
            for i in range(0, a.queries, 1024):
                s = q[i:i + 1024] @ y.t()
                out.append((s > ts[i:i + 1024, None].to(s.dtype)).sum(1))
            return torch.cat(out)
        ms = timed(torch_counts, max(a.iters // 3, 1))
        print(f"torch.mm + compare + sum (1024-query slices): {ms * 1e3:9.1f} us")
    K.check_status(status)


if __name__ == "__main__":
    main()

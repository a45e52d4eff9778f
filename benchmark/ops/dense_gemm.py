"""Dense GEMMs (by default QKV and o_proj + residual of the Mixtral shape) against cuBLAS, with a sweep over kernels and tiles.

    python benchmark/ops/dense_gemm.py [--tokens 64,128,256,512] [--shapes 4096x14336,12288x4096] [--gate] [--sweep]

Every measurement is one CUDA graph of 24 launches over 24 distinct weight matrices (so weights always come from HBM,
as in a decoder stack, and host launch overhead is excluded), timed with CUDA events around graph replays, best of 4.
cuBLAS goes through ``torch.matmul`` / ``torch.addmm`` in the same harness (not with ``--gate``, a SwiGLU product). ``--sweep`` also
tries what the rules of ``ops/gemm.py`` choose from and prints the four fastest: every token tile (32..256) and split-K factor (1..8)
of gemm.cu, every tile width (128..256 weight rows) of the pairs of gemm_wide.cu, and even cuts of the tokens with 1..8 CTAs per cluster of
gemm_split.cu; the last two are what ``dense_wide`` and ``split_plan`` were fitted to.
"""
import argparse
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__)))))

import torch

from disagmoe_b200.ops import gemm

N_WEIGHTS = 24


def bench(fn, n=N_WEIGHTS, reps=4):
    for i in range(n):
        fn(i)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for i in range(n):
            fn(i)
    for _ in range(12):      # clocks and caches settle before anything is timed
        g.replay()
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.replay()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / n * 1e3)
    return best


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--tokens", default="64,128,256,512")
    ap.add_argument("--shapes", help="output x input features, instead of the two of the Mixtral shape")
    ap.add_argument("--gate", action="store_true", help="gated products (of --shapes): two matrices of these sizes")
    ap.add_argument("--sweep", action="store_true")
    ap.add_argument("--tp", type=int, default=1, help="shapes of one rank of a tensor-parallel attention group: QKV has "
                    "6144 / tp output features, o_proj 4096 / tp input features and no residual (reduce-scatter epilogue)")
    ap.add_argument("--hbm-gbs", type=float, default=6549.0, help="copy bandwidth for the weight-streaming floor")
    a = ap.parse_args(argv)
    dev = "cuda"
    shapes = (("qkv", 6144, 4096, False), ("o_proj+residual", 4096, 4096, True)) if a.tp == 1 else \
        ((f"qkv/tp{a.tp}", 6144 // a.tp, 4096, False), (f"o_proj/tp{a.tp}", 4096, 4096 // a.tp, False))
    if a.gate and not a.shapes:
        ap.error("--gate needs --shapes")
    if a.shapes:
        shapes = [(s, *map(int, s.split("x")), False) for s in a.shapes.split(",")]
    for name, F, K, resid in shapes:
        ws = [torch.randn(F * (2 if a.gate else 1), K, device=dev, dtype=torch.bfloat16) * 0.02 for _ in range(N_WEIGHTS)]
        for T in (int(t) for t in a.tokens.split(",")):
            x = torch.randn(T, K, device=dev, dtype=torch.bfloat16)
            r = torch.randn(T, F, device=dev, dtype=torch.bfloat16) if resid else None
            out = torch.empty(T, F, device=dev, dtype=torch.bfloat16)

            def lib(i):
                if resid:
                    torch.addmm(r, x, ws[i].T, out=out)
                else:
                    torch.matmul(x, ws[i].T, out=out)

            def own(i, **kw):
                if a.gate:
                    gemm.swiglu_linear(x, ws[i], out=out, **kw)
                else:
                    gemm.linear(x, ws[i], residual=r, out=out, **kw)

            t_own = bench(own)
            line = (f"{name} T={T}: this kernel {t_own:.1f} us, " + ("" if a.gate else f"cuBLAS {bench(lib):.1f} us, ") +
                    f"weight-streaming floor {ws[0].numel() * 2 / a.hbm_gbs / 1e3:.1f} us")
            if a.sweep:
                tries = [dict(wide=cols) for cols in (128, 160, 192, 224, 256)]
                tries += [dict(bn=bn, wide=False, **({} if a.gate else dict(splitk=sk))) for bn in (32, 64, 128, 256) if bn <= max(32, T)
                          for sk in ((1,) if a.gate else (1, 2, 3, 4, 6, 8))]
                cuts = {-(-(-(-T // n)) // 16) * 16 for n in range(-(-T // 256), -(-T // 16) + 1)}
                tries += [dict(bn=bn, cluster=s) for bn in sorted(cuts) for s in range(1, 9)]
                res = []
                for kw in tries:
                    try:
                        res.append((bench(lambda i: own(i, **kw)), str(kw)))
                    except RuntimeError:      # refused: the first, eager launch says so
                        pass
                res.sort()
                line += "; fastest: " + ", ".join(f"{t:.1f} us {kw}" for t, kw in res[:4])
            print(line, flush=True)
    assert gemm.check_status() == 0


if __name__ == "__main__":
    main()

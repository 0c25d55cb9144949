"""Per-phase device timeline of one decode step.

    python litert-lm_b200/decode_timeline.py [--model gemma3-1b] [--mode 2] [--prompt 1024]

Prints, for every phase class (qkv, attention, o-proj, gate/up, down, head, arg-max), the
time the slowest CTA worked, the barrier latency seen by the last CTA to arrive, and their
sum over the step.  Built on B200Lm_TraceDecodeStep.
"""
from __future__ import annotations

import argparse
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import __graft_entry__ as graft  # noqa: E402


def summarise(stamps: np.ndarray, khz: int, n_layers: int):
    """stamps [n_barriers, n_cta, 2] -> rows (phase, work_max_us, work_mean_us, barrier_us)."""
    nb = stamps.shape[0]
    arrive, release = stamps[:, :, 0].astype(np.float64), stamps[:, :, 1].astype(np.float64)
    us = 1e3 / khz
    work = np.zeros_like(arrive)
    work[1:] = arrive[1:] - release[:-1]
    work[0] = np.nan                      # phase 0 includes kernel start-up
    wait = release - arrive
    names = []
    for _ in range(n_layers):
        names += ["qkv", "attention", "o-proj", "gate/up", "down"]
    names += ["head", "arg-max"]
    rows = {}
    for b in range(nb):
        r = rows.setdefault(names[b], [0.0, 0.0, 0.0, 0])
        if b > 0:
            r[0] += np.nanmax(work[b]) * us
            r[1] += np.nanmean(work[b]) * us
        r[2] += wait[b].min() * us
        r[3] += 1
    return rows


def summarise_chained(pts: np.ndarray, n_layers: int) -> None:
    """Chain of step kernels: pts [n_kernels, n_cta, 8] in nanoseconds: 0 start, 1 predecessor complete,
    2 activations ready, 3 products done, 4 end; zero where a CTA had no part in the kernel."""
    p = pts.astype(np.float64) / 1e3
    names = ["qkv", "attention", "o-proj", "gate/up", "down"] * n_layers + ["head"]
    rows = {}
    for b in range(1, len(names)):
        q, prev = p[b][p[b][:, 4] > 0], p[b - 1][:, 4].max()
        rows.setdefault(names[b], []).append([(q[:, 0] - prev).mean(), (q[:, 1] - prev).mean(), (q[:, 2] - q[:, 1]).mean(), (q[:, 3] - q[:, 2]).mean(),
                                              (q[:, 4] - q[:, 3]).mean(), q[:, 4].max() - prev, len(q)])
    print("us, mean over CTAs and layers, from the end of the previous kernel")
    print(f"{'kernel':10s} {'count':>5s} {'start':>7s} {'released':>9s} {'prologue':>9s} {'products':>9s} {'tail':>6s} {'in all':>7s} {'CTAs':>6s}")
    for name, v in rows.items():
        m = np.mean(v, axis=0)
        print(f"{name:10s} {len(v):5d} {m[0]:7.2f} {m[1]:9.2f} {m[2]:9.2f} {m[3]:9.2f} {m[4]:6.2f} {m[5]:7.2f} {m[6]:6.0f}")
    print(f"step {p[len(names) - 1][:, 4].max() - p[0][:, 0][p[0][:, 0] > 0].min():.1f} us (with the stamps)")


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--model", default="gemma3-1b")
    ap.add_argument("--mode", type=int, default=0)
    ap.add_argument("--prompt", type=int, default=1024)
    args = ap.parse_args()
    sys.path.insert(0, ROOT)
    import bench
    graft.build()
    pkg = graft.load_package()
    cfg, rec, img = bench.load_model(args.model)
    ex = pkg.B200LlmExecutor(img, decode_mode=args.mode)
    ids = np.random.Generator(np.random.PCG64(cfg.seed)).integers(0, cfg.vocab, args.prompt).astype(np.int32)
    ex.Prefill(ids)
    for _ in range(3):
        ex.Decode()
    tok, stamps, khz = ex.TraceDecodeStep()
    if ex.GetDecodeMode() in (pkg.DECODE_CHAINED, pkg.DECODE_PHASE_KERNELS):
        summarise_chained(ex.last_trace_points, cfg.n_layers)
        return
    rows = summarise(stamps, khz, cfg.n_layers)
    total = 0.0
    print(f"model={cfg.name} mode={args.mode} n_cta={stamps.shape[1]} barriers={stamps.shape[0]} sm_clock_khz={khz}")
    print(f"{'phase':10s} {'count':>5s} {'slowest-CTA work us':>20s} {'mean-CTA work us':>17s} {'barrier us':>11s} {'per-phase us':>13s}")
    for name, (wmax, wmean, bar, n) in rows.items():
        total += wmax + bar
        print(f"{name:10s} {n:5d} {wmax:20.1f} {wmean:17.1f} {bar:11.1f} {(wmax + bar) / n:13.2f}")
    print(f"step total (work of slowest CTA + barrier latency): {total:.1f} us")
    pts = getattr(ex, "last_trace_points", None)
    if pts is not None and pts.any():
        names = []
        for _ in range(cfg.n_layers):
            names += ["qkv", "attention", "o-proj", "gate/up", "down"]
        names += ["head", "arg-max"]
        us = 1e3 / khz
        points = [0, 1, 3, 4, 5, 6]           # stamps taken by the streaming kernel (2 is unused)
        labels = ["wait staged", "prologue", "mma", "epilogue", "tail rounds"]
        print("segments inside a phase, mean over CTAs that reached both points (us):")
        for cls in ["qkv", "attention", "o-proj", "gate/up", "down", "head"]:
            idx = [b for b in range(1, len(names)) if names[b] == cls]
            seg = []
            rel = stamps[[b - 1 for b in idx], :, 1].astype(np.float64)
            p = pts[idx].astype(np.float64)
            first = np.where(p[:, :, 0] > 0, (p[:, :, 0] - rel) * us, np.nan)
            seg.append(("release->start", np.nanmean(first)))
            for k in range(len(points) - 1):
                lo, hi = points[k], points[k + 1]
                ok = (p[:, :, lo] > 0) & (p[:, :, hi] > 0)
                d = np.where(ok, (p[:, :, hi] - p[:, :, lo]) * us, np.nan)
                seg.append((labels[k], float(np.nanmean(d)) if ok.any() else float("nan")))
            inner = (((1, 2, "stage q/k/v"), (2, 7, "append + ranges"), (7, 3, "scores"), (3, 5, "P.V"), (5, 6, "reduce + write partials"))
                     if cls == "attention" else ((1, 2, "loads+sums"), (2, 7, "block reduce"), (7, 3, "quantize")))
            for lo, hi, nm in inner:
                ok = (p[:, :, lo] > 0) & (p[:, :, hi] > 0)
                if ok.any():
                    seg.append((nm, float(np.nanmean(np.where(ok, (p[:, :, hi] - p[:, :, lo]) * us, np.nan)))))
            arr = stamps[idx, :, 0].astype(np.float64)
            lastp = np.where(p[:, :, 6] > 0, (arr - p[:, :, 6]) * us, np.nan)
            seg.append(("end->arrive", float(np.nanmean(lastp)) if np.isfinite(lastp).any() else float("nan")))
            print(f"  {cls:10s} " + "  ".join(f"{n}={v:.2f}" for n, v in seg))


if __name__ == "__main__":
    main()

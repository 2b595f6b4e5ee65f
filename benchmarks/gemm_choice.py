"""Times every form of the plain GEMM over a grid of sizes, beside the one that is chosen.

    python benchmarks/gemm_choice.py [--launches 20] > table.md

Operands in L2, launches back to back, CUDA events around ``--launches`` of them; the smaller of two
such times.  One row of markdown per size: the chosen form and its time, the fastest form and its
time, and the times of all forms that apply.  Forms as ``psdev_gemm_config`` names them: 1000 S + BN
one 128 x BN tile per cluster of S CTAs, 2256 / 2512 tiles of pairs of CTAs, 128 persistent one-CTA
tiles."""
import argparse
import math
import os
import sys

import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from ps_lite_b200 import _lib  # noqa: E402
from ps_lite_b200.ops.gemm import gemm_status, linear_bf16  # noqa: E402

ROWS = (64, 128, 256, 512, 1024, 1536, 2048, 4096)
COLS = (256, 512, 1024, 2048, 4096)
SMS = 148


def forms(m, n, k):
    out = [128]
    for bn in (64, 128):
        for split in (1, 2, 4, 8):
            ctas = math.ceil(m / 128) * math.ceil(n / bn) * split
            if split == 1 or (ctas <= 2 * SMS and split <= math.ceil(k / 64)):
                out.append(1000 * split + bn)
    return out + ([2256, 2512] if m >= 256 and n >= 256 else [])


def timed(fn, launches):
    best = math.inf
    for _ in range(3):   # (the first one warms up)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(launches):
            fn()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / launches * 1e3)
    return best


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--launches", type=int, default=20)
    args = ap.parse_args()
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    lib = _lib.device_lib()
    print("| M x N x K | chosen | us | fastest | us | chosen / fastest | all forms, us |")
    print("|---|---|---|---|---|---|---|")
    worst, logs = 1.0, []
    for m in ROWS:
        for n in COLS:
            for k in COLS:
                x = torch.randn(m, k, device=dev).to(torch.bfloat16)
                w = (torch.randn(n, k, device=dev) / k ** 0.5).to(torch.bfloat16)
                out = torch.empty(m, n, device=dev, dtype=torch.bfloat16)
                us = {}
                for form in forms(m, n, k):
                    _lib.check(lib.psdev_gemm_config(form), "psdev_gemm_config")
                    us[form] = timed(lambda: linear_bf16(x, w, out), args.launches)
                _lib.check(lib.psdev_gemm_config(0), "psdev_gemm_config")
                assert gemm_status(dev) == 0
                pick = lib.psdev_gemm_choice(m, n, k) or 128
                best = min(us, key=us.get)
                ratio = us[pick] / us[best]
                worst, _ = max(worst, ratio), logs.append(math.log(ratio))
                each = ", ".join(f"{f}: {t:.1f}" for f, t in us.items())
                print(f"| {m} x {n} x {k} | {pick} | {us[pick]:.1f} | {best} | {us[best]:.1f} | "
                      f"{ratio:.2f} | {each} |", flush=True)
    print(f"\n{len(logs)} sizes: chosen over fastest {math.exp(sum(logs) / len(logs)):.3f} "
          f"(geometric mean), {worst:.2f} at most")


if __name__ == "__main__":
    main()

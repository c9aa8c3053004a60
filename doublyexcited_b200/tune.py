"""The matvec autotuner: ``python -m doublyexcited_b200.tune``.

For every grid (NN = 2N+1) and storage (complex128, complex64) it times one
block matvec with each candidate of one pass -- a kernel family and a cap
on resident CTAs per SM -- the other pass held at its built-in choice,
keeps the fastest per pass -- the built-in choice, the line kernels, unless
another is at least 2 % faster, so that timing noise does not move the
table -- and writes the table that problem handles read
at creation (``matvec_tuning.txt`` beside the library, or ``--out``):

    <storage> <NN> <pass> <family> <ctas_per_sm> <ms_per_vector>

Families: ``ev`` even/odd-split lines in registers (CUDA cores, every grid),
``dmma`` FP64 tensor cores, ``stream`` streaming / cube CUDA-core kernels,
``tf32`` tcgen05 TF32 tensor cores (complex64).  Candidates a grid does not
build fall back to another family inside the library, so they are skipped
here.  What is timed is one product: a table that names another family for a
pass also switches off the exchange-symmetric products and half-vector sums
of the solves that use that pass, which only the line kernels' products keep
exact, and they are worth more than a few percent of a product.  Timing: CUDA
events on the handle's stream, a block of vectors larger than L2 (at least
256 MB), 2 warm-up and 5 timed matvecs per candidate, median of 3 rounds.
"""
from __future__ import annotations

import argparse
import os
import statistics
import sys

# grids each family builds (the library's *_supported functions); the line
# kernels serve every grid and are listed first on these, last on larger ones
# (tune() times them on all)
EV = {"c128": range(9, 14, 2), "c64": range(9, 18, 2)}
EV_LAST = range(15, 24, 2)
DMMA = range(9, 20, 2)
TF32 = range(9, 16, 2)
STREAM_PERSISTENT = range(13, 20, 2)  # smaller grids run the non-persistent cube kernels
FAMILY_CODE = {"ev": "fma", "dmma": "tensor", "stream": "stream", "tf32": "tf32"}
MARGIN = 0.02  # a candidate replaces the built-in choice only when this much faster


BUILT_IN = ("ev", 0)  # what a handle without a table runs, on every grid


def candidates(storage: str, nn: int):
    out = []
    if nn in EV[storage]:
        out.append(("ev", 0))
    out += [("stream", c) for c in ((0, 1) if nn in STREAM_PERSISTENT else (0,))]
    if nn in DMMA:
        out.append(("dmma", 0))
    if storage == "c64" and nn in TF32:
        out += [("tf32", 0), ("tf32", 1)]
    if nn in EV_LAST and nn not in EV[storage]:
        out.append(("ev", 0))
    return out


def time_matblock(torch, prob, storage, x, y, nvec, reps=5):
    call = prob.matblock32_d if storage == "c64" else prob.matblock_d
    for _ in range(2):
        call(x.data_ptr(), y.data_ptr(), nvec)
    rounds = []
    for _ in range(3):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            call(x.data_ptr(), y.data_ptr(), nvec)
        e1.record()
        torch.cuda.synchronize()
        rounds.append(e0.elapsed_time(e1) / reps / nvec)
    return statistics.median(rounds)


def pick(results):
    """The entry of [(ms, family, ctas)] to keep: the built-in choice, or the
    fastest where that is more than MARGIN faster."""
    fastest = min(results)
    built_in = next((r for r in results if r[1:] == BUILT_IN), None)
    return fastest if built_in is None or fastest[0] < (1.0 - MARGIN) * built_in[0] else built_in


def tune(ns, out_path, log=print):
    import torch

    import doublyexcited_b200 as de

    lines = ["# storage NN pass family ctas_per_sm ms_per_vector  (python -m doublyexcited_b200.tune; B200)"]
    for n in ns:
        nn = 2 * n + 1
        for storage in ("c128", "c64"):
            prec = "mixed" if storage == "c64" else "fp64"
            with de.Problem(n=n, delta=2.0, theta=0.3, precision=prec) as prob:
                st = torch.cuda.current_stream()
                prob.set_stream(st.cuda_stream)
                dt = torch.complex64 if storage == "c64" else torch.complex128
                vec_bytes = prob.dim * (8 if storage == "c64" else 16)
                nvec = max(2, min(16, -(-(256 << 20) // vec_bytes)))
                gen = torch.Generator(device="cuda").manual_seed(nn)
                x = torch.randn(nvec, prob.dim, dtype=dt, device="cuda", generator=gen)
                y = torch.empty_like(x)
                best = {}
                for pass_ in (0, 1):
                    prob.set_matvec_kernel("fma")  # the other pass at its built-in choice
                    for p2 in (0, 1):
                        if p2 != pass_ and p2 in best:
                            prob.set_matvec_launch(storage, p2, FAMILY_CODE[best[p2][0]], best[p2][1])
                    res = []
                    for fam, ctas in dict.fromkeys([BUILT_IN] + candidates(storage, nn)):
                        prob.set_matvec_launch(storage, pass_, FAMILY_CODE[fam], ctas)
                        ms = time_matblock(torch, prob, storage, x, y, nvec)
                        res.append((ms, fam, ctas))
                        log(f"  {storage} NN={nn} pass {'AB'[pass_]} {fam:6s} ctas={ctas}  {ms:.4f} ms/vector")
                    ms, fam, ctas = pick(res)
                    best[pass_] = (fam, ctas, ms)
                for pass_ in (0, 1):
                    fam, ctas, ms = best[pass_]
                    lines.append(f"{storage} {nn} {'AB'[pass_]} {fam} {ctas} {ms:.4f}")
                    log(f"{storage} NN={nn} pass {'AB'[pass_]}: {fam} ctas={ctas}")
                del x, y
    with open(out_path, "w") as f:
        f.write("\n".join(lines) + "\n")
    return lines


def main(argv=None):
    ap = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    ap.add_argument("--n", type=int, nargs="*", default=[4, 5, 6, 7, 8, 9],
                    help="grid parameters N (NN = 2N+1) to tune")
    ap.add_argument("--out", default=None, help="table path (default: matvec_tuning.txt beside the library)")
    a = ap.parse_args(argv)
    from . import _lib

    out = a.out or os.path.join(os.path.dirname(_lib.lib_path()), "matvec_tuning.txt")
    # time the candidates, not a table left from an earlier run
    os.environ["DE_MATVEC_TUNING"] = ""
    tune(a.n, out)
    print(f"wrote {out}")
    return 0


if __name__ == "__main__":
    sys.exit(main())

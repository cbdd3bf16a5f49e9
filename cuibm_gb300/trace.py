"""Per-phase times of the linear solves, from the timer stamps they write.

With the option "trace_solve" on, block 0 of a persistent solve stamps the global
timer at every grid barrier together with the source line of the barrier's call
site (include/cuibm.h, CUIBM_F_SOLVE_TRACE).  The time between two stamps is the
phase that ended at the second barrier (its work, its wait for the slowest block
and the barrier itself), so summing by call site shows where a solve spends its
time without a profiler.  A separable solve stamps after each of its kernels instead,
with a line of csrc/separable.cu whose comment names the phase; its phases hold the
stamp's own launch too.  Solves launched phase by phase (fused_solve 0, a hierarchy
without the body's rows) write no stamps.

    python -m cuibm_gb300.trace CASE_FOLDER [--warm 20] [--system poisson] [--flags "-saStructured 0"]

runs the case for --warm steps, traces the next step and prints, per site, the count,
total and mean phase time.
"""
import argparse
import collections
import os

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc")
SEPARABLE = 0x8000  # this bit of a site: a line of separable.cu


def site_text(site):
    """(file:line, the line's text) of a stamp's site."""
    name, line = ("separable.cu", site - SEPARABLE) if site & SEPARABLE else ("fused_kernels.cuh", site)
    path = os.path.join(CSRC, name)
    src = open(path).read().split("\n") if os.path.exists(path) else []
    text = src[line - 1].strip() if 0 < line <= len(src) else ""
    return "%s:%d" % (name, line), text[:60]


def phases(trace):
    """(site line, microseconds) of every phase of one solve's trace."""
    k = int(trace[0])
    e = np.asarray(trace[1:k + 1], dtype=np.uint64)
    ts = (e & np.uint64(0xFFFFFFFFFFFF)).astype(np.int64)
    site = (e >> np.uint64(48)).astype(np.int64)
    dt = np.diff(ts) / 1000.0
    return list(zip(site[1:].tolist(), dt.tolist()))


def table(trace):
    """Per call site: [count, total us], in decreasing total."""
    agg = collections.OrderedDict()
    for line, us in phases(trace):
        a = agg.setdefault(line, [0, 0.0])
        a[0] += 1
        a[1] += us
    return sorted(agg.items(), key=lambda kv: -kv[1][1])


def main(argv=None):
    import cuibm_gb300 as cb
    ap = argparse.ArgumentParser(description=__doc__.split("\n")[0])
    ap.add_argument("case")
    ap.add_argument("--warm", type=int, default=20)
    ap.add_argument("--system", choices=["velocity", "poisson", "both"], default="both")
    ap.add_argument("--flags", default="", help="the solver's command-line flags, e.g. \"-saStructured 0\"")
    ap.add_argument("--sequence", type=int, default=0, metavar="N",
                    help="also list the solve's phases N to 2N in order (one iteration's worth)")
    a = ap.parse_args(argv)
    with cb.NavierStokesSolver(a.case, a.flags.split()) as s:
        s.set_option("write_output", 0)
        s.initialise()
        s.stepTime(a.warm)
        s.set_option("trace_solve", 1)
        s.stepTime(1)
        tr = s.get("solve_trace")
        s.set_option("trace_solve", 0)
        it = s.iterations()
        i = s.info
        print("case %s: %d x %d, SA levels %d, iterations (velocity, Poisson) %s at step %d" % (
            a.case, i.nx, i.ny, i.amg_levels, it, s.timeStep - 1))
        half = len(tr) // 2
        for name, t in (("velocity", tr[:half]), ("poisson", tr[half:])):
            if a.system not in (name, "both"):
                continue
            ph = phases(t)
            if not ph:
                print("%s solve: no stamps (it is launched phase by phase)" % name)
                continue
            total = sum(us for _, us in ph)
            print("%s solve: %d phases, %.1f us" % (name, len(ph), total))
            for line, (n, us) in table(t):
                at, text = site_text(line)
                print("  %-22s  n %4d  total %9.1f us  mean %7.2f us  %5.1f %%  %s" % (
                    at, n, us, us / n, 100 * us / max(total, 1e-9), text))
            if a.sequence:
                print("  phases %d-%d in order:" % (a.sequence, 2 * a.sequence - 1))
                for k, (line, us) in enumerate(ph[a.sequence:2 * a.sequence]):
                    print("    %4d  %-22s  %7.2f us" % (a.sequence + k, site_text(line)[0], us))


if __name__ == "__main__":
    main()

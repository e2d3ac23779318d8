"""Summarise a sweep timestamp trace written by the engine.

Setting ``CCDB_TRACE_FILE=<path>`` makes libccdb trace a fit's sweeps, each findMode
attempt over the one before.  Of a windowed sweep, the default, the file holds CTA
0's SM clock at three points of the first 4,096 rounds and what the round did;
``python -m ccd_b200.trace --rounds <path> [sm_mhz]`` prints where a round's time
goes and how many columns it takes.  Of a grid-wide level sweep it holds, for the
first sweep, the schedule (segments, tasks) and per CTA segment the
global timer at: wait start, level open, end of the CTA-wide phase, end of
the warp phase, arrival.  ``python -m ccd_b200.trace <path>`` prints where the
time of a sweep goes: level-to-level detection, per-level span, and the phase
breakdown by segment kind.

``CCDB_BATCH_TRACE_FILE=<path>`` does the same for mixed-precision batched fits,
which then run the lockstep engine: CTA 0's SM clock at six points of every column of one sweep
(``CCDB_BATCH_TRACE_SWEEP``, default 1).  ``python -m ccd_b200.trace --batch
<path> [sm_mhz]`` prints the per-phase breakdown.
"""
from __future__ import annotations

import sys

import numpy as np

SEG = np.dtype([("level", "i4"), ("n_chunk", "i4"), ("n_cta", "i4"), ("n_warp", "i4"), ("t0", "i8")])
TASK = np.dtype([("col", "i4"), ("kind", "i2"), ("warp", "i2"), ("chunk", "i4"), ("nchunks", "i4"),
                 ("part_base", "i4"), ("p0", "i4"), ("p1", "i4"), ("pad", "i4")])


def load(path: str):
    raw = open(path, "rb").read()
    ns, nt = np.frombuffer(raw[:16], np.int64)
    off = 16
    segs = np.frombuffer(raw[off:off + SEG.itemsize * ns], SEG)
    off += SEG.itemsize * ns
    rest = len(raw) - off - TASK.itemsize * nt - 40 * ns
    G = rest // 8 - 1
    cta_seg = np.frombuffer(raw[off:off + 8 * (G + 1)], np.int64)
    off += 8 * (G + 1)
    tasks = np.frombuffer(raw[off:off + TASK.itemsize * nt], TASK)
    off += TASK.itemsize * nt
    allt = np.frombuffer(raw[off:], np.uint64).astype(np.int64)
    return segs, cta_seg, tasks, allt[:3 * ns].reshape(-1, 3), allt[3 * ns:5 * ns].reshape(-1, 2)


def summarise(path: str) -> str:
    segs, cta_seg, tasks, tr, tr2 = load(path)
    ns = len(segs)
    t0 = tr[tr[:, 0] > 0, 0].min()
    tr = tr - t0
    tr2 = np.where(tr2 > 0, tr2 - t0, 0)
    L = segs["level"]
    nl = int(L.max()) + 1
    first = np.full(nl, 1 << 62)
    last = np.zeros(nl, np.int64)
    for i in range(ns):
        first[L[i]] = min(first[L[i]], tr[i, 1])
        last[L[i]] = max(last[L[i]], tr[i, 2])
    gap = first[1:] - last[:-1]
    span = last - first
    out = [f"segments {ns}, tasks {len(tasks)}, CTAs {len(cta_seg) - 1}, levels {nl}",
           f"sweep span {last[-1] / 1e3:.1f} us, {last[-1] / 1e3 / nl:.2f} us per level",
           f"level-to-level detection: median {np.median(gap) / 1e3:.2f} us",
           f"level span (open -> last arrival): median {np.median(span) / 1e3:.2f} us, "
           f"p90 {np.percentile(span, 90) / 1e3:.2f} us"]
    p1 = tr2[:, 0] - tr[:, 1]
    p2 = np.where(tr2[:, 1] > 0, tr2[:, 1] - tr2[:, 0], 0)
    p3 = tr[:, 2] - np.maximum(tr2[:, 0], tr2[:, 1])
    kinds = (("CTA-task segments", (segs["n_cta"] > 0) & (segs["n_warp"] == 0) & (segs["n_chunk"] == 0)),
             ("warp-only segments", (segs["n_warp"] > 0) & (segs["n_cta"] == 0) & (segs["n_chunk"] == 0)),
             ("split-column segments", segs["n_chunk"] > 0))
    for name, sel in kinds:
        if sel.sum():
            out.append(f"{name}: {int(sel.sum())}, median phase1 {np.median(p1[sel]) / 1e3:.2f} us, "
                       f"phase2 {np.median(p2[sel]) / 1e3:.2f} us, tail {np.median(p3[sel]) / 1e3:.2f} us")
    return "\n".join(out)


ROUND = np.dtype([(n, "i8") for n in ("begin", "steps", "end", "base", "flying", "taken", "moved", "alone")])


def summarise_rounds(path: str, sm_mhz: float = 1965.0) -> str:
    t = np.fromfile(path, ROUND)
    t = t[t["end"] != 0]
    us = 1.0 / sm_mhz
    cycle = np.flatnonzero(np.diff(t["base"]) < 0)
    out = [f"rounds traced: {len(t)}, cycles ended: {len(cycle)}; columns taken {int(t['taken'].sum())}, "
           f"moved {int(t['moved'].sum())}; {t['taken'].mean():.2f} taken of {t['flying'].mean():.2f} in flight a round"]
    for name, sel in (("several columns", t["alone"] == 0), ("one column alone", t["alone"] != 0)):
        s = t[sel]
        if not len(s):
            continue
        moves = s["moved"] > 0
        out.append(f"  {name}: {len(s)} rounds, median {np.median(s['end'] - s['begin']) * us:.2f} us: to the steps "
                   f"{np.median(s['steps'] - s['begin']) * us:.2f}, to the end "
                   f"{np.median((s['end'] - s['steps'])[moves]) * us if moves.any() else 0:.2f} where one moves, "
                   f"{np.median((s['end'] - s['steps'])[~moves]) * us if (~moves).any() else 0:.2f} where none does")
    return "\n".join(out)


BATCH_PHASES = ("issue (stage, prefetch, metadata)", "gather + FP32 terms", "group reduction",
                "step + update", "cp.async wait + barrier")


def summarise_batch(path: str, sm_mhz: float = 1965.0) -> str:
    tr = np.fromfile(path, np.int64).reshape(-1, 6)
    cols = np.nonzero(tr[:, 0])[0]
    t = tr[cols]
    per = np.diff(t, axis=1)  # five phases
    span = np.diff(t[:, 0])
    us = 1.0 / sm_mhz
    out = [f"columns traced: {len(cols)}; sweep span {(t[-1, 5] - t[0, 0]) * us / 1e3:.2f} ms; "
           f"median column {np.median(span) * us:.2f} us (mean {span.mean() * us:.2f} us)"]
    for name, col in zip(BATCH_PHASES, per.T):
        out.append(f"  {name:34s} median {np.median(col) * us:7.3f} us  mean {col.mean() * us:7.3f} us  "
                   f"share {col.sum() / per.sum():6.1%}")
    return "\n".join(out)


if __name__ == "__main__":
    if sys.argv[1] == "--batch":
        print(summarise_batch(sys.argv[2], *(float(a) for a in sys.argv[3:4])))
    elif sys.argv[1] == "--rounds":
        print(summarise_rounds(sys.argv[2], *(float(a) for a in sys.argv[3:4])))
    else:
        print(summarise(sys.argv[1]))

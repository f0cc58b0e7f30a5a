"""The stage kernel's whole named-barrier sequence, simulated on the CPU for every compiled variant
under several schedules.

Per tile (bbdg_stage_fast_impl.cuh), element warps of group g `bar.sync` the group's B->A barrier
(tiles after the first), its A->B barrier and, with more than one warp per element, the group's
trace barrier, which only the group's own threads count towards; chain warps `bar.sync` every
group's B->A barrier (tiles after the first), then `bar.arrive` on every group's A->B barrier. A
barrier phase completes when its own count of threads has arrived; threads of two phases must not
mix, and every warp must finish.
"""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "bernsteinbasis.jl_gb300", "csrc")


def read(name):
    with open(os.path.join(CSRC, name)) as fh:
        return fh.read()


def variants():
    return [(int(n), p, int(e), int(t)) for n, p, e, t in
            re.findall(r"X\((\d+), (BB_WAVE|BB_MAXWELL), (\d+), (\d+)\)",
                       read("bbdg_stage_fast_variants.h"))]


def program(EPB, TPE, NCH, T):
    """Each warp's list of (sync or arrive, barrier), and the thread count of every barrier."""
    CHT = (EPB * 4 * NCH + 31) // 32 * 32
    GS = 1 if EPB <= 7 else (EPB + 6) // 7
    NG = EPB // GS
    assert EPB % GS == 0 and TPE % 32 == 0
    ids = 3 * NG if TPE > 32 else 2 * NG
    assert ids <= 15, "named barriers 1..15"
    count = {b: GS * TPE + CHT for b in range(1, 2 * NG + 1)}
    count.update({b: GS * TPE for b in range(2 * NG + 1, 3 * NG + 1)})
    warps = []
    for w in range(EPB * TPE // 32):
        g = (w * 32 // TPE) // GS
        ops = []
        for it in range(T):
            if it > 0:
                ops.append(("sync", 1 + NG + g))
            ops.append(("sync", 1 + g))
            if TPE > 32:
                ops.append(("sync", 1 + 2 * NG + g))
        warps.append(ops)
    for _ in range(CHT // 32):
        ops = []
        for it in range(T):
            if it > 0:
                ops += [("sync", 1 + NG + g) for g in range(NG)]
            ops += [("arrive", 1 + g) for g in range(NG)]
        warps.append(ops)
    return warps, count


def finishes(warps, count, pick):
    pc = [0] * len(warps)
    arrived, waiting = {}, {}
    ready = set(range(len(warps)))
    while ready:
        w = pick(sorted(ready))
        if pc[w] >= len(warps[w]):
            ready.discard(w)
            continue
        kind, b = warps[w][pc[w]]
        arrived[b] = arrived.get(b, 0) + 32
        if arrived[b] > count[b]:
            return False
        pc[w] += 1
        if kind == "sync":
            waiting.setdefault(b, []).append(w)
            ready.discard(w)
        if arrived[b] == count[b]:
            arrived[b] = 0
            ready.update(waiting.pop(b, []))
    return all(p >= len(ops) for p, ops in zip(pc, warps)) and not any(arrived.values())


def test_the_sequence_is_the_kernels():
    """The barrier instructions of the kernel, in its order."""
    code = read("bbdg_stage_fast_impl.cuh")
    body = code[code.index("stage_fast_kernel(FastStageParams P)"):]
    used = re.findall(r"(nbar_sync|nbar_arrive)\(([^;]*?)\)[;,]", body)
    assert used == [("nbar_sync", "1 + NG + g, GCOUNT"), ("nbar_arrive", "1 + g, GCOUNT"),
                    ("nbar_sync", "1 + NG + grp, GCOUNT"), ("nbar_sync", "1 + grp, GCOUNT"),
                    ("nbar_sync", "1 + 2 * NG + grp, L::GS * TPE")]
    assert "TRACE_SMEM = TPE > 32" in code and "GCOUNT = GS * TPE + CHT" in code


@pytest.mark.parametrize("tiles", [1, 2, 5])
def test_every_variant_finishes(tiles):
    vs = variants()
    assert len(vs) >= 20
    for N, phys, EPB, TPE in vs:
        warps, count = program(EPB, TPE, 2 if phys == "BB_WAVE" else 6, tiles)
        rng = random.Random(N * 100 + tiles)
        for pick in (lambda r: r[0], lambda r: r[-1], rng.choice):
            assert finishes(warps, count, pick), (N, phys, EPB, TPE)


def test_a_missing_arrival_is_seen():
    """Without one warp's trace barrier the simulation does not finish."""
    warps, count = program(4, 64, 2, 3)
    last = [i for i, op in enumerate(warps[0]) if op[1] > 8][-1]
    del warps[0][last]
    assert not finishes(warps, count, lambda r: r[0])

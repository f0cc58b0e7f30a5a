"""Generates bbdg_lift_slots.cuh: where the FP32 lift keeps entry q of a face's stack.

A warp's lanes gather 32 consecutive coefficients n from the four face stacks of an element at
the positions of the permutations of src/BernsteinLift.jl:207-218. In volume order up to five of
the 32 entries fall into one shared-memory bank. Which slot of the stack an entry occupies is
free: every chain writes its own stack with the same slot in every lane, and the stacks' odd
stride spreads the lanes over the banks. So each entry is given a slot such that, in every group
and face, few entries share a bank: simulated annealing over swaps, seeded, one table per degree.

  python gen_lift_slots.py > bbdg_lift_slots.cuh
"""
import multiprocessing as mp

import numpy as np

DEGREES = (6, 7, 8, 9, 11)
SWEEPS = 30000  # swap attempts per entry


def tables(N):
    idx = [(i, j, k) for k in range(N + 1) for j in range(N + 1 - k) for i in range(N + 1 - k - j)]
    at = {a: m for m, a in enumerate(idx)}
    reads = []
    for i, j, k in idx:
        l = N - i - j - k  # noqa: E741
        reads.append([at[(i, k, j)], at[(j, k, l)], at[(j, k, i)], at[(i, j, k)]])
    return np.array(reads)


def wavefronts(slot, reads):
    """Shared-memory wavefronts of one element's gather."""
    tot = 0
    for g in range(0, len(reads), 32):
        for f in range(4):
            tot += np.bincount(slot[reads[g:g + 32, f]] % 32, minlength=32).max()
    return int(tot)


def anneal(N):
    reads = tables(N)
    NP = len(reads)
    groups = (NP + 31) // 32
    edge = np.zeros((NP, 4), int)  # the (face, group) in which entry q is read
    for f in range(4):
        edge[reads[:, f], f] = np.arange(NP) // 32
    rng = np.random.default_rng(N)
    slot = np.arange(NP)
    bank = [int(b) for b in slot % 32]
    cnt = [[[0] * 32 for _ in range(groups)] for _ in range(4)]
    ed = edge.tolist()
    for q in range(NP):
        for f in range(4):
            cnt[f][ed[q][f]][bank[q]] += 1
    steps = SWEEPS * NP
    best, best_slot = wavefronts(slot, reads), slot.copy()
    for it in range(steps):
        if it % 65536 == 0:
            qs = rng.integers(NP, size=65536).tolist()
            rs = rng.integers(NP, size=65536).tolist()
            us = rng.random(65536).tolist()
            temp = max(0.05, 1.0 - 1.1 * it / steps)
            w = wavefronts(slot, reads)
            if w < best:
                best, best_slot = w, slot.copy()
        q, r = qs[it % 65536], rs[it % 65536]
        bq, br = bank[q], bank[r]
        if bq == br:
            continue
        d = 0
        for f in range(4):
            eq, er = ed[q][f], ed[r][f]
            if eq != er:
                cq, cr = cnt[f][eq], cnt[f][er]
                d += cq[br] - cq[bq] + cr[bq] - cr[br] + 2
        if d <= 0 or us[it % 65536] < np.exp(-d / temp):
            for f in range(4):
                eq, er = ed[q][f], ed[r][f]
                cnt[f][eq][bq] -= 1
                cnt[f][eq][br] += 1
                cnt[f][er][br] -= 1
                cnt[f][er][bq] += 1
            bank[q], bank[r] = br, bq
            slot[q], slot[r] = slot[r], slot[q]
    w = wavefronts(slot, reads)
    if w < best:
        best, best_slot = w, slot.copy()
    return N, wavefronts(np.arange(NP), reads), best, 4 * groups, best_slot.tolist()


def main():
    with mp.get_context("spawn").Pool() as pool:
        res = pool.map(anneal, DEGREES[::-1], chunksize=1)
    print('''// Generated by gen_lift_slots.py; do not edit. Entry q of a degree-N face stack lives at slot
// lift_slot<N>(q) (see the generator for how the slots were chosen).
#pragma once
#include <stdint.h>

template <int N>
__host__ __device__ __forceinline__ constexpr int lift_slot(int q) {
  return q;
}
// The same at run time, from device memory.
template <int N>
__device__ __forceinline__ int lift_slot_at(int q) {
  return q;
}''')
    for N, ident, best, ideal, slot in sorted(res):
        print(f'''
// N = {N}: {best} wavefronts per element's gather ({ident} in volume order, {ideal} without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<{N}>(int q) {{
  switch (q) {{''')
        moved = [f"case {q}: return {v};" for q, v in enumerate(slot) if v != q]
        for a in range(0, len(moved), 4):
            print("    " + " ".join(moved[a:a + 4]))
        print('''    default: return q;
  }
}''')
        print(f"static __device__ const uint16_t lift_slots_{N}[{len(slot)}] = {{")
        for a in range(0, len(slot), 20):
            print("    " + ", ".join(str(v) for v in slot[a:a + 20]) + ",")
        print(f'''}};
template <>
__device__ __forceinline__ int lift_slot_at<{N}>(int q) {{
  return lift_slots_{N}[q];
}}''')


if __name__ == "__main__":
    main()

#!/usr/bin/env python3
"""Generate row_tables.inc: the sector order of the N <= 8 stage kernel.

An ADO (N x N complex) is stored as P = N(N-1)/2 + ceil(N/2) sectors of
32 B; each sector holds a symmetric pair (w(i,j), w(j,i)) or two diagonal
elements.  The kernel runs one warp per ADO; lane (r, t) = 4r + t holds the
sectors of the pairs {r, 2t} and {r, 2t+1} (the diagonal sector in place of
{r, r}): they are its operands of the commutator, and what it reads of the
neighbours along the baths of state r.  A sector is held by two lanes; one of
them owns it and writes it, and its first half is the element of the owner's
row (the first of the two diagonal elements).

The sectors owned by row r lie side by side, row after row: a warp's store of
an ADO is linear in its lanes (8 wavefronts of the L1 against 22 when the
sectors are permuted), and the owned sectors of a neighbour's row are one
128-byte line for N = 8.  Within a row this script searches (simulated
annealing) the order of the sectors, so that the four operand reads of a
quarter warp -- row and column element of either sector -- hit different
16-byte bank groups.  The result is deterministic for the fixed seeds below.

Usage: python gen_row_tables.py OUT.inc
"""
import math
import random
import sys
from collections import Counter


def col_owned(r, t):
    """Which of its two sectors (0: {r, 2t}, 1: {r, 2t+1}) lane (r, t) owns."""
    R = r >> 1
    return 0 if t == R else (r & 1) ^ (1 if R > t else 0)


def sectors(n):
    """Per sector its two elements (first, second), owner's row first."""
    out = []
    for r in range(n):
        for t in range(4):
            c = 2 * t + col_owned(r, t)
            if c >= n:
                continue
            if c == r:
                out.append(((r, r), (min(r + 1, n - 1),) * 2))
            else:
                out.append(((r, c), (c, r)))
    return out


def reads(n):
    """Quarter-warp operand reads: lists of (sector, half)."""
    secs = sectors(n)
    where = {}
    for k, (a, b) in enumerate(secs):
        where.setdefault(a, (k, 0))
        where.setdefault(b, (k, 1))
    out = []
    for R in range(4):
        for s in range(2):
            for which in range(2):
                group = []
                for r in (2 * R, 2 * R + 1):
                    for t in range(4):
                        c = 2 * t + s
                        if r >= n or c >= n:
                            continue
                        k, h = where[(r, c)]
                        if which == 1:
                            if r != c:
                                k, h = where[(c, r)]
                            elif s == 0:
                                h = 1  # the second diagonal element (the lane's own output needs it)
                        group.append((k, h))
                if group:
                    out.append(group)
    return secs, out


def conflicts(groups, perm):
    c = 0
    for g in groups:
        hit = {}
        for k, h in g:
            hit.setdefault((2 * perm[k] + h) % 8, set()).add((k, h))
        c += max(len(v) for v in hit.values()) - 1
    return c


def search(n, iters):
    secs, groups = reads(n)
    rows = {}
    for k, (x, _) in enumerate(secs):
        rows.setdefault(x[0], []).append(k)
    best = None
    for seed in range(4):
        rng = random.Random(100 * n + seed)
        perm = list(range(len(secs)))  # sectors() lists them row by row
        cur = conflicts(groups, perm)
        if best is None or cur < best[0]:
            best = (cur, perm[:])
        movable = [r for r in rows if len(rows[r]) > 1]
        for it in range(iters if movable else 0):
            T = 2.0 * (1 - it / iters) ** 2 + 0.01
            a, b = rng.sample(rows[rng.choice(movable)], 2)
            perm[a], perm[b] = perm[b], perm[a]
            new = conflicts(groups, perm)
            if new <= cur or rng.random() < math.exp((cur - new) / T):
                cur = new
                if cur < best[0]:
                    best = (cur, perm[:])
            else:
                perm[a], perm[b] = perm[b], perm[a]
    table = [None] * len(secs)
    for k in range(len(secs)):
        table[best[1][k]] = secs[k]
    return table, best[0]


def main():
    e1, e2 = ["    {0},"], ["    {0},"]
    for n in range(1, 9):
        table, conf = search(n, 40000)
        a = ", ".join(str(x[0] * n + x[1]) for x, _ in table)
        b = ", ".join(str(y[0] * n + y[1]) for _, y in table)
        e1.append("    {%s}, /* N=%d extra wavefronts=%d */" % (a, n, conf))
        e2.append("    {%s}," % b)
        print(n, conf, file=sys.stderr, flush=True)
    with open(sys.argv[1], "w") as f:
        f.write("/* Generated by gen_row_tables.py: sector order of the N <= 8 stage kernel.\n"
                " * kRowE1[N][p], kRowE2[N][p] = row-major element index of the two halves of\n"
                " * sector p (equal for the padding half of an odd N's last diagonal sector). */\n")
        f.write("static const signed char kRowE1[9][32] = {\n" + "\n".join(e1) + "\n};\n")
        f.write("static const signed char kRowE2[9][32] = {\n" + "\n".join(e2) + "\n};\n")


if __name__ == "__main__":
    main()

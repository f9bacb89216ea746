"""CPU restatement of the plain walk's rounds and term list (plain_walk in
pot_walk.cu): which node each lane takes, what a round appends to the list,
and when whole 32-entry lists are evaluated."""
from __future__ import annotations

import numpy as np

LEVELS = 21
PW_CAP = 640
PW_RESERVE = 7 * (LEVELS + 1)
LIST = 64  # entries the list holds


def tree(x, w):
    """Leaf-size-1 octree of points x in [0, w]^3 as nested nodes:
    ("cell", centre, width, children), ("part", i) or ("bucket", [i, ...]), the
    last a cell of the deepest level that holds several particles."""
    dig = np.zeros((len(x), LEVELS), int)
    lo, hi = np.zeros_like(x), np.full_like(x, w)
    for l in range(LEVELS):
        mid = (lo + hi) * 0.5
        up = x >= mid
        dig[:, l] = up[:, 0] * 4 + up[:, 1] * 2 + up[:, 2]
        lo, hi = np.where(up, mid, lo), np.where(up, hi, mid)

    def make(members, level):
        if len(members) == 1:
            return ("part", int(members[0]))
        if level == LEVELS:
            return ("bucket", members.tolist())
        kids = []
        for d in range(8):
            m = members[dig[members, level] == d]
            if len(m):
                kids.append(make(m, level + 1))
        return ("cell", x[members].mean(0), w / 2 ** level, kids)

    return make(np.arange(len(x)), 0)


def walk(root, x, targets, theta, flush_before_buckets=True):
    """One warp's walk for the particles `targets`.  Returns (largest list
    index written, entries in evaluation order as (entry, targets' mask))."""
    pts = [x[t] for t in targets]
    stack = [(root, (1 << len(targets)) - 1)]
    take, lst, done, high = 1, [], [], -1

    def flush():
        nonlocal lst
        done.extend(lst[:32])
        lst = lst[32:64]  # the entries beyond the first 32 move to the front

    def put(entry):
        nonlocal high
        lst.append(entry)
        high = max(high, len(lst) - 1)

    while stack or take:
        nodes = [stack.pop() for _ in range(take)]
        opened, buckets = [], []
        for node, mask in nodes:
            if node[0] == "cell":
                acc = 0
                for k, p in enumerate(pts):
                    if node[2] ** 2 < theta ** 2 * ((p - node[1]) ** 2).sum():
                        acc |= 1 << k
                if mask & ~acc:
                    opened.append((node[3], mask & ~acc))
                if mask & acc:
                    put((("cell", tuple(node[1])), mask & acc))
            elif node[0] == "part":
                m = mask & ~sum(1 << k for k, t in enumerate(targets) if t == node[1])
                if m:
                    put((("part", node[1]), m))
            else:
                buckets.append((node[1], mask))
        for kids, m in opened:
            stack.extend((c, m) for c in kids)
        for members, mask in buckets:
            for j0 in range(0, len(members), 32):
                if flush_before_buckets and len(lst) >= 32:
                    flush()
                for j in members[j0:j0 + 32]:
                    put((("part", j), mask & ~sum(1 << k for k, t in enumerate(targets) if t == j)))
                if not flush_before_buckets and len(lst) >= 32:
                    flush()
        take = min(len(stack), 32)
        if len(stack) + 7 * take > PW_CAP - PW_RESERVE:
            take = max(1, min(take, (PW_CAP - PW_RESERVE - len(stack)) // 7))
        assert len(stack) <= PW_CAP
        if len(lst) >= 32:
            flush()
    done.extend(lst)
    return high, done

"""CPU: the sector order of the N <= 8 stage kernel (row_tables.inc): every
element once, a sector's first half in its owner's row, the sectors of a row
side by side -- what the kernel's lanes take for granted."""
import os
import re

import pytest


def tables(root):
    text = open(os.path.join(root, "dm-heom_b200", "csrc", "row_tables.inc")).read()
    out = []
    for name in ("kRowE1[9]", "kRowE2[9]"):
        body = text[text.index(name):]
        body = re.sub(r"/\*.*?\*/", "", body[body.index("= {"):body.index("};")])
        out.append([[int(v) for v in re.findall(r"\d+", row)] for row in re.findall(r"\{([\d,\s]+)\}", body)])
    return out


def owned(r, t):  # row_owned of heom_kernels.cuh
    return 0 if t == r // 2 else (r & 1) ^ (1 if r // 2 > t else 0)


@pytest.mark.parametrize("n", range(1, 9))
def test_row_order(root, n):
    e1, e2 = (t[n] for t in tables(root))
    assert len(e1) == len(e2) == n * (n - 1) // 2 + (n + 1) // 2
    cells = [e for a, b in zip(e1, e2) for e in ({a, b})]
    assert sorted(cells) == list(range(n * n))
    rows = []
    for a, b in zip(e1, e2):
        (r, c), (r2, c2) = divmod(a, n), divmod(b, n)
        if r == c:
            assert r % 2 == 0 and (r2, c2) == (min(r + 1, n - 1),) * 2
        else:
            assert (r2, c2) == (c, r)
        assert c == 2 * (c // 2) + owned(r, c // 2)
        rows.append(r)
    assert rows == sorted(rows)

"""The order of reads and writes of the exact fold's window lists
(csrc/smc_coop.cuh, fold_grid), on the CPU.

A tile writes its list, all tiles exchange, then each reads every tile's list;
the next fold may follow at once.  Every interleaving of the tiles is walked
through: no tile may read a list that a later fold has rewritten.  The number of
list sets is the source's; with one set the walk finds the overwritten list, so it
can tell.
"""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def source_sets():
    text = open(os.path.join(ROOT, "mckl_b200", "csrc", "smc_coop.cuh")).read()
    fold = text[text.index("bool fold_grid("):]
    fold = fold[:fold.index("void seg_fold(")]
    m = re.search(r"constexpr unsigned kWinSets = (\d+);", text)
    if not m:
        return 1
    # one choice of the set per fold, and no list reached past it
    assert len(re.findall(r"\+\+c\.folds % kWinSets", fold)) == 1 and fold.count("c.g.win") == 1
    return int(m.group(1))


def overwritten(tiles, folds, sets):
    """Whether some interleaving has a tile read a list that is not its fold's.
    A tile's program: per fold a write, a publish, a wait for every publish, and
    a read of each tile's list."""
    ops = []
    for n in range(folds):
        ops += [("write", n), ("publish", n), ("await", n)] + [("read", n, t) for t in range(tiles)]
    start = ((0,) * tiles, (0,) * tiles, ((-1,) * sets,) * tiles)  # positions, publishes, list contents
    seen, todo = {start}, [start]
    while todo:
        pos, pub, lists = todo.pop()
        for t in range(tiles):
            if pos[t] == len(ops):
                continue
            op = ops[pos[t]]
            p, li = pub, lists
            if op[0] == "write":
                mine = list(lists[t])
                mine[op[1] % sets] = op[1]
                li = lists[:t] + (tuple(mine),) + lists[t + 1:]
            elif op[0] == "publish":
                p = pub[:t] + (op[1] + 1,) + pub[t + 1:]
            elif op[0] == "await":
                if min(pub) < op[1] + 1:
                    continue
            elif lists[op[2]][op[1] % sets] != op[1]:
                return True
            nxt = (pos[:t] + (pos[t] + 1,) + pos[t + 1:], p, li)
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
    return False


@pytest.mark.parametrize("tiles,folds", [(2, 6), (3, 3)])
def test_no_list_is_rewritten_while_it_is_read(tiles, folds):
    assert overwritten(tiles, folds, 1)
    assert not overwritten(tiles, folds, source_sets())

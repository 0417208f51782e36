"""The roles of a CTA meet through barriers whose phases are waited for by parity.  Such a wait holds as long as the phase
after the one that is meant cannot complete before it has been looked at: then the parity has turned back and the wait blocks.
Here the roles run as models on the CPU, each made of the waits and arrivals of its kernel, with any one or two of them held up
for as long as the others can go on.  Whatever is held up, every role ends, and no wait passes before its phase is complete."""
import itertools
import re
from collections import deque
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "self-forcing_b200" / "csrc"


class Barrier:
    def __init__(self, count=1):
        self.count = self.pending = count
        self.phase = 0                                   # the phase that is not complete yet

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.phase, self.pending = self.phase + 1, self.count


def run(roles, engines, held):
    """Steps the roles (generators of waits (barrier, phase), or None between two actions) and the engines (queues of
    completions).  Those in `held` move only when nothing else can, one action at a time.  Returns who did not end."""
    waits = {name: None for name in roles}

    def step(name):
        if name in engines:
            if engines[name]:
                engines[name].popleft()()
                return True
            return False
        if name not in waits:
            return False
        if waits[name] is not None:
            bar, phase = waits[name]
            if (bar.phase ^ phase) & 1 == 0:             # as mbarrier.test_wait.parity sees it
                return False
            assert bar.phase > phase, f"{name}: passed before its phase was complete"
        try:
            waits[name] = next(roles[name])
        except StopIteration:
            del waits[name]
        return True

    free = [n for n in [*roles, *engines] if n not in held]
    while True:
        moved = False
        for name in free:
            while step(name):
                moved = True
        if not moved and not any(step(name) for name in held):
            return sorted(waits)


def never_stuck(build):
    names = [*build()[0], *build()[1]]
    for held in [(), *((n,) for n in names), *itertools.permutations(names, 2)]:
        left = run(*build(), held)
        assert not left, f"with {held} held up: {left} never end"


def row_backward(F, wants_kv, n_rt, n_k, n_dr, units=2):
    """monarch_bwd_row_tc_kernel: `wants_kv[i]` steps give dK / dV; n_rt row tiles, n_k K tiles, n_dr barriers for dR."""
    one = lambda n, count=1: [Barrier(count) for _ in range(n)]
    q_full, v_full, v_empty, s_full, rz_free, dkv_full, dkv_free = one(7)
    q_empty, s_read, dr_read, r_full, p_full = one(5, 2)
    k_full, k_empty, rt_full, rt_empty = one(n_k), one(n_k), one(n_rt), one(n_rt)
    dr_full, dq_full, dq_free = one(n_dr), one(2), one(2)
    eng = {n: deque() for n in ("rows", "tiles", "sdr", "grad")}      # copies in order, GEMMs of the two issuing warps
    steps = [(u, i, u * F + i) for u in range(units) for i in range(F)]
    rt = lambda g, which: divmod(2 * g + which, n_rt)                  # uses of the slot before this one, slot

    def load_rows():
        for _, _, g in steps:
            for which in range(2):
                use, s = rt(g, which)
                yield rt_empty[s], use - 1
                eng["rows"].append(rt_full[s].arrive)

    def load_tiles():
        for u, i, g in steps:
            if i == 0:
                yield q_empty, u - 1
                eng["tiles"].append(q_full.arrive)
            yield k_empty[g % n_k], g // n_k - 1
            eng["tiles"].append(k_full[g % n_k].arrive)
            yield v_empty, g - 1
            eng["tiles"].append(v_full.arrive)

    def issue_sdr():
        for u, i, g in steps:
            if i == 0:
                yield q_full, u
            yield k_full[g % n_k], g // n_k
            yield s_read, g - 1
            eng["sdr"].append(s_full.arrive)
            if i + 1 == F:
                eng["sdr"].append(q_empty.arrive)
            yield dr_read, g - 1
            for which in range(2):
                use, s = rt(g, which)
                yield rt_full[s], use
                if which:
                    yield v_full, g
                if not wants_kv[i]:
                    eng["sdr"].append(rt_empty[s].arrive)
            eng["sdr"] += [dr_full[g % n_dr].arrive, v_empty.arrive]

    def issue_grad():
        gd = 0
        last = max([i for i in range(F) if wants_kv[i]], default=0)
        for u, i, g in steps:
            if wants_kv[i]:
                yield r_full, gd
                yield None
                yield dr_full[g % n_dr], g // n_dr
                yield dkv_free, gd - 1
                eng["grad"] += [rt_empty[rt(g, 0)[1]].arrive, rt_empty[rt(g, 1)[1]].arrive]
            yield p_full, g
            if i == 0:
                yield dq_free[u & 1], (u >> 1) - 1
            eng["grad"].append(k_empty[g % n_k].arrive)
            if wants_kv[i]:
                eng["grad"].append(dkv_full.arrive)
                gd += 1
            if i == last:
                eng["grad"].append(q_empty.arrive)
            eng["grad"].append(rz_free.arrive)
            if i + 1 == F:
                eng["grad"].append(dq_full[u & 1].arrive)

    def elementwise():
        for _, i, g in steps:
            yield s_full, g
            s_read.arrive()
            yield rz_free, g - 1
            if wants_kv[i]:
                r_full.arrive()
                yield None
            yield dr_full[g % n_dr], g // n_dr
            dr_read.arrive()
            yield None
            p_full.arrive()

    def drain():
        gd = 0
        for u in range(units + 1):
            for i in range(F if u < units else 0):
                if wants_kv[i]:
                    yield dkv_full, gd
                    dkv_free.arrive()
                    gd += 1
            if u:
                yield dq_full[(u - 1) & 1], (u - 1) >> 1
                dq_free[(u - 1) & 1].arrive()

    return {"load_rows": load_rows(), "load_tiles": load_tiles(), "issue_sdr": issue_sdr(), "issue_grad": issue_grad(),
            "elementwise0": elementwise(), "elementwise1": elementwise(), "drain": drain()}, eng


@pytest.mark.parametrize("wants_kv", ["1111", "1100", "0110", "0001", "0000", "1"])
def test_row_backward(wants_kv):
    text = (CSRC / "monarch_bwd_row_tc.cu").read_text()
    slots = int(re.search(r"kRowSlots = (\d+);", text).group(1))
    n_dr = int((re.search(r"uint64_t[^;]*\bdr_full\[(\d+)\]", text) or [0, 1])[1])
    kv = [c == "1" for c in wants_kv]
    for n_rt in range(3, slots + 1):
        for n_k in (2, 3):
            never_stuck(lambda: row_backward(len(kv), kv, n_rt, n_k, n_dr))


def column_step(groups, tiles, units, n_q, n_a, n_y, first):
    """monarch_l_tc_kernel: groups of `units` units with tiles[group] key tiles, n_q query tiles, n_a / n_y slots for key and
    value tiles; the warp of the value tiles waits for the barrier `first` before its first load."""
    one = lambda n: [Barrier() for _ in range(n)]
    q_full, q_empty, cl_full, cl_empty = one(n_q), one(n_q), one(4), one(4)
    a_full, a_empty, y_full, y_empty = one(n_a), one(n_a), one(n_y), one(n_y)
    s_full, p_full, sp_free, o_full, o_free = one(2), one(2), one(2), one(2), one(2)
    named = {"q_full[0]": q_full[0], "q_first": Barrier()}
    eng = {n: deque() for n in ("keys", "values", "queries", "s", "pv")}
    order = [(gi, t) for gi in range(groups) for t in range(tiles[gi])]

    def load_keys():
        x = 0
        for gt in range(len(order)):
            for _ in range(units):
                yield a_empty[x % n_a], x // n_a - 1
                eng["keys"].append(a_full[x % n_a].arrive)
                x += 1
            yield cl_empty[gt & 3], (gt >> 2) - 1
            eng["keys"].append(cl_full[gt & 3].arrive)

    def load_values():
        for x in range(len(order) * units):
            yield y_empty[x % n_y], x // n_y - 1
            if x == 0 and first:
                yield named[first], 0
            eng["values"].append(y_full[x % n_y].arrive)

    def issue_s():
        x = gt = 0
        for step in range(groups + n_q - 1):
            if step < groups:
                yield q_empty[step % n_q], step // n_q - 1
                eng["queries"].append(q_full[step % n_q].arrive)
            gi = step - (n_q - 1)
            if gi < 0:
                continue
            yield q_full[gi % n_q], gi // n_q
            if gi == 0:
                named["q_first"].arrive()
            for _ in range(tiles[gi]):
                yield sp_free[gt & 1], (gt >> 1) - 1
                for _ in range(units):
                    yield a_full[x % n_a], x // n_a
                    eng["s"].append(a_empty[x % n_a].arrive)
                    x += 1
                eng["s"].append(s_full[gt & 1].arrive)
                gt += 1
            eng["s"].append(q_empty[gi % n_q].arrive)

    def issue_pv():
        x, used = 0, [0, 0]
        for gt, (gi, t) in enumerate(order):
            w = gt & 1
            yield p_full[w], gt >> 1
            if t < 2:
                yield o_free[w], used[w] - 1
                used[w] += 1
            for _ in range(units):
                yield y_full[x % n_y], x // n_y
                eng["pv"].append(y_empty[x % n_y].arrive)
                x += 1
            eng["pv"].append(sp_free[w].arrive)
            if t + 1 == tiles[gi]:
                eng["pv"].append(o_full[gi & 1].arrive)

    def softmax(w):
        used = 0
        for gt, (gi, t) in enumerate(order):
            if gt & 1 != w:
                continue
            yield s_full[w], gt >> 1
            yield cl_full[gt & 3], gt >> 2
            cl_empty[gt & 3].arrive()
            if t + 2 >= tiles[gi]:
                yield o_free[w], used - 1
                used += 1
            p_full[w].arrive()

    def epilogue():
        gt = 0
        for gi in range(groups):
            yield o_full[gi & 1], gi >> 1
            o_free[gt & 1].arrive()
            if tiles[gi] > 1:
                o_free[gt & 1 ^ 1].arrive()
            gt += tiles[gi]

    return {"load_keys": load_keys(), "load_values": load_values(), "issue_s": issue_s(), "issue_pv": issue_pv(),
            "softmax0": softmax(0), "softmax1": softmax(1), "epilogue": epilogue()}, eng


@pytest.mark.parametrize("tiles", [[1], [2], [3], [5], [1, 2, 3]], ids=str)
@pytest.mark.parametrize("units,n_q", [(1, 2), (2, 2), (4, 1), (4, 2)])
def test_column_step(units, n_q, tiles):
    text = (CSRC / "monarch_lstep_tc.cu").read_text()
    first = re.search(r"mbar_wait_u\(&bars->(q_\w+(?:\[0\])?), 0\)\)", text)
    for n_a, n_y in ((2, 3), (3, 5)):
        never_stuck(lambda: column_step(6, (tiles * 6)[:6], units, n_q, n_a, n_y, first and first.group(1)))

"""CPU: the hand-overs of the pair-row sigma kernel
(pyscf-forge_b200/csrc/sigma_mp.cu), restated and run under random schedules,
and its shares of a job table.

Hand-overs: two stages each of D (movers to MMA warps) and V (back), every one
an mbarrier with the kernel's counts and parities, and the named barrier of
the movers.  No schedule deadlocks, an MMA warp reads D of its own tile from
every mover, a mover scatters V of its own tile from every MMA warp, and no
buffer is overwritten before its last reader.

Shares: the CTAs' tiles of all rounds make up the list exactly, and the jobs
that a CTA poisons when a hand-over was lost are those it has had tiles of."""
import random

import pytest


class _Mbar:
    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passes(self, parity):  # mbarrier.try_wait.parity
        return (self.phase & 1) != parity


def _mma(n):
    for it in range(n):
        s, ph = it & 1, (it >> 1) & 1
        yield ("wait", "Dfull", s, ph)
        yield ("read", "D", s, it)
        yield ("arrive", "Dempty", s)
        if it >= 2:
            yield ("wait", "Vempty", s, ph ^ 1)
        yield ("write", "V", s, it)
        yield ("arrive", "Vfull", s)


def _mover(columns):
    it0 = 0
    for m in columns:  # mp_movers: a column tile of a job
        end = it0 + m
        for it in range(it0, end + 1):
            if it < end:
                s = it & 1
                if it >= 2:
                    yield ("wait", "Dempty", s, ((it >> 1) & 1) ^ 1)
                yield ("write", "D", s, it)
                yield ("arrive", "Dfull", s)
            if it > it0:
                s = (it - 1) & 1
                yield ("wait", "Vfull", s, ((it - 1) >> 1) & 1)
                yield ("read", "V", s, it - 1)
                yield ("arrive", "Vempty", s)
            yield ("bar",)
        it0 = end


def _run(columns, nmma, nmov, seed):
    rng = random.Random(seed)
    n = sum(columns)
    bars = {k: [_Mbar(c) for _ in range(2)]
            for k, c in (("Dfull", nmov), ("Dempty", nmma), ("Vfull", nmma), ("Vempty", nmov))}
    writers = {"D": nmov, "V": nmma}
    held = {b: [dict() for _ in range(2)] for b in writers}  # part of each writer: the tile it holds
    unread = {b: [0, 0] for b in writers}                    # reads of the present tile still to come
    warps = [_mma(n) for _ in range(nmma)] + [_mover(columns) for _ in range(nmov)]
    cur = [next(w, None) for w in warps]
    at_bar = set()
    while any(c is not None for c in cur):
        ready = [i for i, c in enumerate(cur) if c is not None and i not in at_bar
                 and not (c[0] == "wait" and not bars[c[1]][c[2]].passes(c[3]))]
        assert ready, "deadlock"
        i = rng.choice(ready)
        op = cur[i]
        if op[0] == "bar":
            at_bar.add(i)
            if len(at_bar) == nmov:
                for j in at_bar:
                    cur[j] = next(warps[j], None)
                at_bar = set()
            continue
        if op[0] == "arrive":
            bars[op[1]][op[2]].arrive()
        elif op[0] == "write":
            buf, s, it = op[1:]
            if it not in held[buf][s].values():
                assert unread[buf][s] == 0, ("overwritten before its last reader", buf, it)
                held[buf][s] = {}
                unread[buf][s] = nmma + nmov - writers[buf]
            held[buf][s][i] = it
        elif op[0] == "read":
            buf, s, it = op[1:]
            assert list(held[buf][s].values()) == [it] * writers[buf], ("another tile", buf, it)
            unread[buf][s] -= 1
        cur[i] = next(warps[i], None)
    assert all(u == 0 for v in unread.values() for u in v)


@pytest.mark.parametrize("nmma,nmov", [(4, 12), (8, 12), (12, 12), (2, 3)])
def test_hand_overs(nmma, nmov):
    for columns in ([1], [2], [1, 1, 1], [3, 1, 4], [2, 2, 5, 1], [7], []):
        for seed in range(12):
            _run(columns, nmma, nmov, seed)


def _find(tiles, t):
    """mp_find: job of tile t of the list, and the tile's number in the job."""
    for j0 in range(0, len(tiles), 32):
        upto = 0
        for j in range(j0, min(j0 + 32, len(tiles))):
            if t < upto + tiles[j]:
                return j, t - upto
            upto += tiles[j]
        t -= upto
    return len(tiles) - 1, t


def _shares(tiles, grid, rounds, cta):
    total = sum(tiles)
    for r in range(rounds):
        q = r * grid + cta
        t0 = total * q // (grid * rounds)
        n = total * (q + 1) // (grid * rounds) - t0
        if n:
            yield t0, n


def _worked(tiles, grid, rounds, cta):
    """(job, tile of the job) of every tile, as both roles walk them."""
    out = []
    for t0, n in _shares(tiles, grid, rounds, cta):
        jb, t = _find(tiles, t0)
        while n:
            m = min(n, tiles[jb] - t)
            out += [(jb, t + k) for k in range(m)]
            n, jb, t = n - m, jb + 1, 0
    return out


def _poisoned(tiles, grid, rounds, cta):
    """mp_poison."""
    out = set()
    for t0, n in _shares(tiles, grid, rounds, cta):
        jb, t = _find(tiles, t0)
        while n > 0:
            m = min(n, tiles[jb] - t)
            if m > 0:
                out.add(jb)
            n, jb, t = n - m, jb + 1, 0
    return out


def test_shares_and_poisoned_jobs():
    rng = random.Random(7)
    for _ in range(300):
        tiles = [rng.choice([0, 0, 1, 2, 7, 33, 200]) for _ in range(rng.choice([1, 2, 5, 40, 70]))]
        if not any(tiles):
            tiles[0] = 1
        grid, rounds = rng.choice([1, 3, 148]), rng.choice([1, 2, 7])
        work = [_worked(tiles, grid, rounds, c) for c in range(grid)]
        assert sorted(x for w in work for x in w) == [(j, t) for j, n in enumerate(tiles) for t in range(n)]
        for c, w in enumerate(work):
            assert _poisoned(tiles, grid, rounds, c) == {j for j, _ in w}

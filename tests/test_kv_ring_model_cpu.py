"""Host model of the attention pipeline's bookkeeping (megaattention_b200/csrc/fused_prefill.cu):
the TMA producer, the one MMA issuer of both tiles, the two softmax warpgroups and the store
warp, on mbarriers with phases and parities as the hardware has them, in both stage layouts of
the K/V ring: shared stages (the heads of a task share a kv head: one K and one V tile per key
block) and separate stages (per key block the K tiles of the task's heads, then their V tiles).

Each role is a Python generator that says which barrier it waits for; a random scheduler lets
one go on at a time.  Loads land and MMAs run later than they are issued, at random (MMAs in
order, as the tensor pipe runs them).  Checked in every interleaving: an MMA finds in its slot
the tile that the program means, no load lands in a slot whose readers are not through, and
the pipeline never stops before the last task's last store."""
import random

import pytest

KV_SLOTS = 5


class Bar:
    """mbarrier: ``wait(parity)`` holds once the phase of that parity is complete."""

    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def wait(self, parity):
        return (self.phase & 1) != parity


class Model:
    def __init__(self, tasks, sep, kv_slots, rng, late_k=False):
        self.tasks, self.sep, self.n, self.rng, self.late_k = tasks, sep, kv_slots, rng, late_k
        n = kv_slots
        self.kv_full, self.kv_empty = [Bar(1) for _ in range(n)], [Bar(1) for _ in range(n)]
        self.q_full, self.q_empty = [Bar(1) for _ in range(2)], [Bar(2) for _ in range(2)]
        self.s_full, self.p_full, self.o_staged, self.o_done, self.o_free = (
            [Bar(1) for _ in range(2)] for _ in range(5))
        self.kv, self.q = [None] * n, [None] * 2       # what the buffers hold
        self.readers = [0] * n                         # MMAs issued on a slot, not yet run
        self.loads, self.pipe = [], []                 # in flight
        self.released, self.stored, self.ran = [], [], set()

    # -------------------------------------------------------------- the hardware's side
    def landable(self):
        """Loads that may land now; with ``late_k`` a K tile lands after the P V of the block
        before it (same head) has run."""
        return [x for x in self.loads
                if not (self.late_k and x[0] == "kv" and x[2][2] == 0 and x[2][1] > 0
                        and (x[2][0], x[2][1] - 1, 1, x[2][3]) not in self.ran)]

    def land(self):
        load = self.rng.choice(self.landable())
        self.loads.remove(load)
        what, i, tile = load
        if what == "kv":
            assert self.readers[i] == 0, "a load into a slot that an MMA still reads"
            self.kv[i] = tile
            self.kv_full[i].arrive()
        else:
            self.q[i] = tile
            self.q_full[i].arrive()

    def run_mma(self):
        op = self.pipe.pop(0)
        if op[0] == "commit":
            op[1].arrive()
        else:
            _, slot, kv_tile, i, q_tile = op
            assert self.kv[slot] == kv_tile, (self.kv[slot], kv_tile)
            assert q_tile is None or self.q[i] == q_tile
            self.readers[slot] -= 1
            self.ran.add(kv_tile)

    def mma(self, slot, kv_tile, i=0, q_tile=None):
        self.readers[slot] += 1
        self.pipe.append(("mma", slot, kv_tile, i, q_tile))

    def commit(self, bar):
        self.pipe.append(("commit", bar))

    def release(self, slot, tile):
        self.released.append(tile)
        self.commit(self.kv_empty[slot])

    # -------------------------------------------------------------- the kernel's roles
    def producer(self):
        slot, ph, q_uses = 0, 0, [0, 0]
        for t, (nt, nblk) in enumerate(self.tasks):
            for i in range(nt):
                yield self.q_empty[i], (q_uses[i] & 1) ^ 1
                q_uses[i] += 1
                self.loads.append(("q", i, (t, i)))
            nld = nt if self.sep else 1
            for jj in range(nblk):
                for ld in range(2 * nld):
                    which = int(ld >= nld)                 # 0 = K, 1 = V
                    head = (ld - nld if which else ld) if self.sep else None
                    yield self.kv_empty[slot], ph ^ 1
                    self.loads.append(("kv", slot, (t, jj, which, head)))
                    slot += 1
                    if slot == self.n:
                        slot, ph = 0, ph ^ 1

    def issuer(self):
        pos, n, sep = [0, 0], self.n, self.sep
        q_par, p_par, o_uses = [0, 0], [0, 0], [0, 0]

        def take(per):
            s, p = pos
            pos[0] += per
            if pos[0] >= n:
                pos[0] -= n
                pos[1] ^= 1
            return s, p

        def at(r, i):
            s, p = r
            if sep and i:
                s += 1
                if s == n:
                    s, p = 0, p ^ 1
            return s, p

        for t, (nt, nblk) in enumerate(self.tasks):
            per = nt if sep else 1
            k = take(per)
            for i in range(nt):
                yield self.q_full[i], q_par[i]
                q_par[i] ^= 1
                if i == 0:
                    for x in range(per):
                        s, p = at(k, x)
                        yield self.kv_full[s], p
                ks = at(k, i)[0]
                tile = (t, 0, 0, i if sep else None)
                self.mma(ks, tile, i, (t, i))
                self.commit(self.s_full[i])
                if sep or i == nt - 1:
                    self.release(ks, tile)
                if nblk == 1:
                    self.commit(self.q_empty[i])
            for jj in range(nblk):
                has_next = jj + 1 < nblk
                v = take(per)
                if has_next:
                    k = take(per)
                for i in range(nt):
                    (vs, vp), (ks, kp) = at(v, i), at(k, i)
                    head = i if sep else None
                    v_tile, k_tile = (t, jj, 1, head), (t, jj + 1, 0, head)
                    last_use = sep or i == nt - 1
                    if sep or i == 0 or jj == 0:
                        yield self.kv_full[vs], vp
                        if has_next and not sep:
                            yield self.kv_full[ks], kp
                        if jj == 0:
                            yield self.o_free[i], (o_uses[i] & 1) ^ 1
                            o_uses[i] += 1
                    yield self.p_full[i], p_par[i]
                    p_par[i] ^= 1
                    self.mma(vs, v_tile)
                    if has_next:
                        if sep:                   # the next K tile is not waited for before P V
                            self.release(vs, v_tile)
                            yield self.kv_full[ks], kp
                        self.mma(ks, k_tile, i, (t, i))
                        self.commit(self.s_full[i])
                        if last_use and not sep:
                            self.release(vs, v_tile)
                        if last_use:
                            self.release(ks, k_tile)
                        if jj + 2 == nblk:
                            self.commit(self.q_empty[i])
                    else:
                        self.commit(self.o_done[i])
                        if last_use:
                            self.release(vs, v_tile)

    def softmax(self, i):
        s_par = o_par = 0
        for nt, nblk in self.tasks:
            if i >= nt:
                continue
            for _ in range(nblk):
                yield self.s_full[i], s_par
                s_par ^= 1
                self.p_full[i].arrive()
            yield self.o_done[i], o_par
            o_par ^= 1
            self.o_free[i].arrive()
            self.q[i] = "staged O"
            self.o_staged[i].arrive()

    def store(self):
        par = [0, 0]
        for t, (nt, _) in enumerate(self.tasks):
            for i in range(nt):
                yield self.o_staged[i], par[i]
                par[i] ^= 1
                assert self.q[i] == "staged O"
                self.stored.append((t, i))
                self.q_empty[i].arrive()

    # -------------------------------------------------------------- any interleaving
    def run(self):
        roles = [self.producer(), self.issuer(), self.softmax(0), self.softmax(1), self.store()]
        waits = {}
        for r in roles:
            waits[r] = next(r, None)
        while True:
            can = [r for r, w in waits.items() if w is not None and w[0].wait(w[1])]
            hw = [f for f, q in ((self.land, self.landable()), (self.run_mma, self.pipe)) if q]
            if not can and not hw:
                break
            pick = self.rng.choice(can + hw)
            if pick in waits:
                waits[pick] = next(pick, None)
            else:
                pick()
        assert all(w is None for w in waits.values()), "the pipeline stopped"
        assert self.stored == [(t, i) for t, (nt, _) in enumerate(self.tasks) for i in range(nt)]
        tiles = [(t, jj, which, h) for t, (nt, nblk) in enumerate(self.tasks) for jj in range(nblk)
                 for which in (0, 1) for h in (range(nt) if self.sep else [None])]
        assert sorted(self.released, key=str) == sorted(tiles, key=str)      # each slot, once


def check(tasks, sep, rng, kv_slots=KV_SLOTS):
    Model(tasks, sep, kv_slots, rng).run()


def test_shared_and_separate_stage_rings_stay_consistent():
    rng = random.Random(7)
    for _ in range(60):
        n = rng.randint(1, 8)
        # shared stages: two heads per task, or one; separate: the odd head runs alone
        check([(2, rng.randint(1, 9)) for _ in range(n)], False, rng)
        check([(rng.choice((1, 2, 2)), rng.randint(1, 9)) for _ in range(n)], True, rng)
        check([(1, rng.randint(1, 9)) for _ in range(n)], False, rng)


@pytest.mark.parametrize("sep", [False, True])
def test_one_issuer_releases_every_slot_once(sep):
    rng = random.Random(8)
    for first in (1, 2):
        for blocks in ([1], [1, 1, 1], [2, 1, 3], [5, 4, 1, 1, 2], [9, 1]):
            for _ in range(4):
                check([(2 if sep and i % 2 else first, b) for i, b in enumerate(blocks)], sep, rng)


def test_separate_stages_p_v_does_not_wait_for_the_next_k():
    """With separate stages the ring holds 1.25 key blocks and the next K tile is often late:
    P V goes on without it."""
    rng = random.Random(10)
    for _ in range(20):
        tasks = [(rng.choice((1, 2)), rng.randint(1, 6)) for _ in range(4)]
        Model(tasks, True, KV_SLOTS, rng, late_k=True).run()


def test_the_model_sees_a_ring_that_is_too_short():
    """Shared stages need a V tile and the next K tile at once, separate ones both first K tiles."""
    for sep in (False, True):
        check([(2, 3)], sep, random.Random(9), kv_slots=2)
        with pytest.raises(AssertionError, match="stopped"):
            check([(2, 3)], sep, random.Random(9), kv_slots=1)

"""Host-side model of the barrier protocols of the two pipelined attention kernels (no GPU needed).

`csrc/attention/attn_fwd_dual.cu` and `csrc/attention/attn_bwd_pipe.cu` each run four or five sequential roles (loader, MMA issuers,
softmax groups) that meet on mbarriers and, where the forward's two softmax groups take turns, on two named barriers.  The roles are transcribed here as generators over the same barriers with the
hardware's phase-parity semantics, asynchronous work (TMA copies, tcgen05 products) completes after a random delay, in order per
issuing thread, and a random scheduler interleaves the roles.  The model checks, for every tile geometry the launchers can
produce, that every role finishes (no wait can stay unsatisfied: on the GPU that would be a bounded wait giving up), and that
no buffer is overwritten while a product that reads it is still in flight or before its consumer has taken it.
"""
import random

import pytest


class Barrier:
    """mbarrier: `count` arrivals complete a phase; `done(parity)` is try_wait.parity (true once the phase of that parity is over)."""

    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.phase += 1
            self.pending = self.count

    def done(self, parity):
        return (self.phase & 1) != (parity & 1)


class NamedBarrier:
    """`bar.sync` by one group of 128 threads and `bar.arrive` by another, 256 in all.  Unlike an mbarrier's, the wait has no limit; and a group that
    comes twice before the other has come would complete the barrier by itself."""

    def __init__(self):
        self.here, self.phase = set(), 0

    def arrive(self, group):
        assert group not in self.here, "a group arrives twice in one phase of a named barrier"
        self.here.add(group)
        if len(self.here) == 2:
            self.here.clear()
            self.phase += 1

    def sync(self, group):
        before = self.phase
        self.arrive(group)
        yield self, before

    def done(self, before):
        return self.phase > before


class AsyncQueue:
    """Work issued to an asynchronous unit by one thread: items complete in issue order after a random delay; an item is a
    callable run at completion (a commit's arrival, a copy's arrival, releasing a read lock)."""

    def __init__(self, rng, max_delay):
        self.rng, self.max_delay, self.items = rng, max_delay, []

    def push(self, fn):
        self.items.append([self.rng.randint(0, self.max_delay), fn])

    def tick(self):
        if self.items:
            if self.items[0][0] <= 0:
                self.items.pop(0)[1]()
                return True
            self.items[0][0] -= 1
        return False


def run(roles, queues, rng, limit=400000, starved=None, starve=0.0):
    """Random interleaving of the role generators; each yields (barrier, parity) to wait or None to be rescheduled.
    `starved`: a role that is skipped with probability `starve` each round (a thread that is slow to notice its barrier)."""
    waiting = {name: None for name in roles}
    live = dict(roles)
    for _ in range(limit):
        if not live and not any(q.items for q in queues):
            return
        for q in queues:
            q.tick()
        names = list(live)
        rng.shuffle(names)
        for name in names:
            if name == starved and rng.random() < starve:
                continue
            cond = waiting[name]
            if cond is not None and not cond[0].done(cond[1]):
                continue
            try:
                waiting[name] = next(live[name])
            except StopIteration:
                del live[name]
                waiting[name] = None
    stuck = {n: (id(w[0]), w[1]) for n, w in waiting.items() if n in live and w is not None}
    raise AssertionError(f"roles never finished: {sorted(live)} waiting on {stuck}")


# ---- forward: two query tiles per CTA -------------------------------------------------------------------------------------------

TURN_TILES = 12                             # DU_TURN_TILES in csrc/attention/attn_fwd_dual.cu


def forward_dual(q0, window, seq_len, rng, max_delay, stages=4, starved=None, turns=None, without=None):
    """`turns`: the launcher's choice of the kernel with turns (by the host's window, which may exceed a device-resident one).  `without`: a part
    of the turn protocol that is left out, which has to show."""
    tile = 128
    turns = min(window, seq_len) >= TURN_TILES * tile if turns is None else turns
    first_a, first_b = q0 - window, q0 + tile - window
    lo_a, lo_b = (first_a // tile if first_a > 0 else 0), (first_b // tile if first_b > 0 else 0)
    hi_a = q0 // tile
    total = hi_a + 1 - lo_a + 1
    n = [hi_a - lo_a + 1, hi_a + 1 - lo_b + 1]
    u0 = [0, lo_b - lo_a]
    bar_q = Barrier(1)
    bar_s, bar_p, bar_o = [Barrier(1), Barrier(1)], [Barrier(1), Barrier(1)], [Barrier(1), Barrier(1)]      # bar_p: the 128 threads as one
    bar_full, bar_free = [Barrier(1) for _ in range(stages)], [Barrier(2) for _ in range(stages)]
    tma, mma = AsyncQueue(rng, max_delay), [AsyncQueue(rng, max_delay), AsyncQueue(rng, max_delay)]
    stage_tile = [None] * stages           # key/value tile a stage holds (None while a copy is in flight)
    readers = [0] * stages                 # products in flight that read the stage
    s_owner = ["free", "free"]             # S_x columns: free -> product in flight -> ready for the softmax -> free
    p_ready = [False, False]
    pv_running = [False, False]            # a product in flight reads P_x and accumulates into O_x
    in_turn, my_turn = turns and n[0] >= TURN_TILES, [NamedBarrier(), NamedBarrier()]      # named barriers 1 and 2
    exponentials = [False, False]
    finished = []

    def loader():
        tma.push(bar_q.arrive)
        for u in range(total):
            st, use = u % stages, u // stages
            if use > 0:
                yield bar_free[st], use - 1
            assert readers[st] == 0, "a stage is refilled while a product still reads it"
            stage_tile[st] = None

            def landed(st=st, u=u):
                stage_tile[st] = u
                bar_full[st].arrive()
            tma.push(landed)
        finished.append("loader")

    def issuer(x):
        def issue_s(u):
            st = u % stages
            yield bar_full[st], u // stages
            assert stage_tile[st] == u, "S reads a stage that does not hold its key tile"
            assert s_owner[x] == "free", "S overwrites scores the softmax has not consumed"
            s_owner[x] = "mma"
            readers[st] += 1

            def done(st=st):
                readers[st] -= 1
                s_owner[x] = "ready"
                bar_s[x].arrive()
            mma[x].push(done)

        yield bar_q, 0
        yield from issue_s(u0[x])
        for i in range(n[x]):
            yield bar_p[x], i
            assert p_ready[x], "PV issued before P was written"
            p_ready[x] = False
            st = (u0[x] + i) % stages
            assert stage_tile[st] == u0[x] + i, "PV reads a stage that does not hold its value tile"
            if i + 1 < n[x]:                            # the next tile's S goes first
                yield from issue_s(u0[x] + i + 1)
            assert stage_tile[st] == u0[x] + i, "PV reads a stage that does not hold its value tile"
            readers[st] += 1
            pv_running[x] = True

            def pv_done(st=st):
                readers[st] -= 1
                pv_running[x] = False
                bar_o[x].arrive()
            mma[x].push(pv_done)
        finished.append(f"issuer{x}")

    def softmax(x):
        lo_x = lo_a if x == 0 else lo_b
        if in_turn and x == 1 and without != "first arrival":
            my_turn[0].arrive(1)
        for i in range(n[x]):
            yield bar_s[x], i
            assert s_owner[x] == "ready"
            yield None                                 # the maximum of the row
            if i > 0:
                yield bar_o[x], i - 1
                assert not pv_running[x]
                done = lo_x + i - 1
                fb = bar_free[(done - lo_a) % stages]
                fb.arrive()
                if (done < lo_b) if x == 0 else (done > hi_a):
                    fb.arrive()
            if in_turn and i < n[0]:
                yield from my_turn[x].sync(x)
                exponentials[x] = True
                assert not all(exponentials), "both query tiles at their exponentials in one turn"
            yield None                                 # the arithmetic: other roles run meanwhile
            exponentials[x] = False
            last = n[0] if without == "last turn's rule" else n[0] - 1
            if in_turn and (x == 0 or i < last):
                my_turn[1 - x].arrive(x)
            assert not pv_running[x], "P or O touched while a product still uses them"
            s_owner[x] = "free"
            p_ready[x] = True
            bar_p[x].arrive()
        yield bar_o[x], n[x] - 1
        finished.append(f"softmax{x}")

    roles = {"loader": loader(), "issuer0": issuer(0), "issuer1": issuer(1), "softmax0": softmax(0), "softmax1": softmax(1)}
    run(roles, [tma] + mma, rng, starved=starved, starve=0.95)
    assert len(finished) == 5 and not any(b.here for b in my_turn)


@pytest.mark.parametrize("seq_len,window", [(256, 0), (256, 1000), (512, 128), (768, 77), (1024, 300), (2048, 1024), (2048, 1000), (2048, 5000),
                                            (4096, 4096), (4096, 129)])
@pytest.mark.parametrize("max_delay", [0, 3, 40])
def test_forward_with_two_query_tiles_never_stalls_and_never_reuses_a_live_buffer(seq_len, window, max_delay):
    rng = random.Random(seq_len * 131 + window * 7 + max_delay)
    for q0 in range(0, seq_len, 256):
        for _ in range(3):
            forward_dual(q0, min(window, seq_len), seq_len, rng, max_delay)


@pytest.mark.parametrize("max_delay", [0, 3, 40])
@pytest.mark.parametrize("window", [1535, 1536, 1537, 1663, 1664, 2000, 4096])      # B has as many key tiles as A, or one more; eleven, twelve, thirteen ..
def test_forward_turns_end_for_every_count_of_key_tiles(window, max_delay):
    rng = random.Random(window * 3 + max_delay)
    for q0 in range(1024, 3584, 256):
        for starved in (None, "softmax0", "softmax1", "issuer0", "issuer1"):
            forward_dual(q0, window, 4096, rng, max_delay, starved=starved, turns=True)


@pytest.mark.parametrize("without", ["first arrival", "last turn's rule"])
def test_forward_model_notices_a_turn_that_is_not_passed_on(without):
    for seed in range(5):
        with pytest.raises(AssertionError):
            forward_dual(2048, 2000, 4096, random.Random(seed), 3, without=without)


def test_forward_model_notices_a_ring_that_is_too_shallow():
    """The check has teeth: a ring of one stage cannot serve two query tiles that are one key tile apart (a stage is released only
    when both have finished with it, and the tile ahead needs the next key tile first); the model reports it (as the stall that the kernel would
    report through its status word, or as a product reading a stage that holds another tile).  Two stages already suffice for progress; the kernel uses four for prefetch."""
    with pytest.raises(AssertionError):                # a stall, or a product that finds the wrong tile in the only stage
        forward_dual(1280, 1024, 2048, random.Random(0), 3, stages=1)
    for seed in range(10):
        forward_dual(1280, 1024, 2048, random.Random(seed), 3, stages=2)


# ---- backward: transposed scores, P and dS in TMEM, dQ drained by warps of its own -------------------------------------------------

def backward_pipe(n_iter, rng, max_delay, stages=3, starved=None, without=None):
    """`without`: a wait that is left out, which has to show."""
    one = ("kv", "s", "p", "dv", "dp", "ds", "dk", "mma", "dq", "end")           # many-thread barriers as one arrival
    bar = {name: Barrier(1) for name in one}
    ring = {name: [Barrier(1) for _ in range(stages)] for name in ("qdo", "free", "stat")}
    tma, mma = AsyncQueue(rng, max_delay), AsyncQueue(rng, max_delay)
    stage_iter, readers = [None] * stages, [0] * stages
    stats = [None] * stages
    s_cols, dp_cols = {"state": "free"}, {"state": "free"}      # S; dP, then dS in the same columns
    p_cols = {"holds": None, "reader": False}
    ds_tile = [{"holds": None, "reader": False}, {"holds": None, "reader": False}]
    dq_cols = {"holds": None}
    drained, finished = [], []

    def commit(*names):
        def done():
            for b in names:
                b.arrive()
        mma.push(done)

    def loader():
        tma.push(bar["kv"].arrive)
        for it in range(n_iter):
            st = it % stages
            if it >= stages:
                yield ring["free"][st], it // stages - 1
            assert readers[st] == 0, "a Q/dO stage is refilled while a product still reads it"
            stage_iter[st] = None

            def landed(st=st, it=it):
                stage_iter[st] = it
                ring["qdo"][st].arrive()
            tma.push(landed)
        finished.append("loader")

    def product(st, it, start, done):
        assert stage_iter[st] == it and stats[st] == it, "a product reads a stage that holds another tile"
        start()
        readers[st] += 1

        def complete():
            readers[st] -= 1
            done()
        mma.push(complete)

    def issuer():
        def issue_s(it):
            assert s_cols["state"] == "free", "S overwritten before the softmax warps have read it"
            product(it % stages, it, lambda: s_cols.update(state="mma"), lambda: s_cols.update(state=it))
            commit(bar["s"])

        def issue_dp(it):
            assert dp_cols["state"] == "free", "dP overwrites dS before dK has used it"
            product(it % stages, it, lambda: dp_cols.update(state="mma"), lambda: dp_cols.update(state=it))
            commit(bar["dp"])

        yield bar["kv"], 0
        yield ring["qdo"][0], 0
        yield ring["stat"][0], 0
        issue_s(0)
        issue_dp(0)
        for it in range(n_iter):
            st, nxt, more = it % stages, (it + 1) % stages, it + 1 < n_iter
            yield bar["p"], it
            if more:
                yield ring["qdo"][nxt], (it + 1) // stages
                yield ring["stat"][nxt], (it + 1) // stages
                issue_s(it + 1)
            assert p_cols["holds"] == it
            product(st, it, lambda: p_cols.update(reader=True), lambda: p_cols.update(reader=False))
            commit(bar["dv"])
            yield bar["ds"], it
            assert dp_cols["state"] == ("dS", it) and ds_tile[it & 1]["holds"] == it
            product(st, it, lambda: None, lambda: dp_cols.update(state="free"))
            commit(bar["dk"])
            if it > 0 and without != "dq":
                yield bar["dq"], it - 1
            assert dq_cols["holds"] is None, "dQ overwritten before it was drained"
            ds_tile[it & 1]["reader"] = True

            def dq_done(it=it):
                ds_tile[it & 1]["reader"] = False
                dq_cols["holds"] = it
            mma.push(dq_done)
            commit(ring["free"][st], bar["mma"])
            if more:
                if without != "dk":
                    yield bar["dk"], it
                issue_dp(it + 1)
        commit(bar["end"])
        finished.append("issuer")

    def drain():
        def put(jt):
            stats[jt % stages] = jt
            ring["stat"][jt % stages].arrive()
        for jt in range(min(stages, n_iter)):
            put(jt)
        for jt in range(n_iter):
            yield bar["mma"], jt
            assert dq_cols["holds"] == jt
            yield None
            dq_cols["holds"] = None
            drained.append(jt)
            bar["dq"].arrive()
            if jt + stages < n_iter:
                assert readers[jt % stages] == 0, "statistics replaced while a product still reads them"
                put(jt + stages)
        finished.append("drain")

    def softmax():
        for it in range(n_iter):
            yield ring["stat"][it % stages], it // stages
            yield bar["s"], it
            assert s_cols["state"] == it and stats[it % stages] == it
            yield None                                 # P formed
            if it > 0 and without != "dv":
                yield bar["dv"], it - 1
            assert not p_cols["reader"], "P overwritten while dV still reads it"
            p_cols["holds"] = it
            s_cols["state"] = "free"
            bar["p"].arrive()
            yield bar["dp"], it
            assert dp_cols["state"] == it and stats[it % stages] == it
            yield None                                 # dS formed
            assert not ds_tile[it & 1]["reader"], "dS stored while dQ of two tiles ago still reads it"
            ds_tile[it & 1]["holds"] = it
            dp_cols["state"] = ("dS", it)
            bar["ds"].arrive()
        yield bar["end"], 0
        assert not any(readers) and drained[: n_iter - 1] == list(range(n_iter - 1))
        finished.append("softmax")

    roles = {"loader": loader(), "issuer": issuer(), "drain": drain(), "softmax": softmax()}
    run(roles, [tma, mma], rng, starved=starved, starve=0.95)
    assert len(finished) == 4 and drained == list(range(n_iter))


@pytest.mark.parametrize("n_iter", [1, 2, 3, 4, 5, 9, 18, 36])
@pytest.mark.parametrize("max_delay", [0, 3, 40])
def test_pipelined_backward_never_stalls_and_never_reuses_a_live_buffer(n_iter, max_delay):
    rng = random.Random(n_iter * 17 + max_delay)
    for _ in range(5):
        backward_pipe(n_iter, rng, max_delay)


@pytest.mark.parametrize("broken", [dict(without="dk"), dict(without="dq", starved="drain"), dict(without="dv"), dict(stages=1)])
def test_backward_model_notices_what_is_missing(broken):
    """dP issued before dK has read dS; dQ before a slow drain has taken the last one; P stored before dV has read it; one Q / dO stage."""
    with pytest.raises(AssertionError):
        for seed in range(20):
            backward_pipe(9, random.Random(seed), 40, **broken)


@pytest.mark.parametrize("starved", ["loader", "issuer0", "issuer1", "softmax0", "softmax1"])
def test_forward_protocol_survives_a_role_that_lags_far_behind(starved):
    """A role that notices its barriers late (so that a barrier it waits on may have moved on by more than one phase where the
    protocol allows that) only delays the others; parity tests never mistake a later phase for an earlier one."""
    rng = random.Random(sum(map(ord, starved)))
    for q0 in (0, 256, 1280, 1792):
        forward_dual(q0, 1024, 2048, rng, 5, starved=starved)


@pytest.mark.parametrize("starved", ["loader", "issuer", "drain", "softmax"])
def test_backward_protocol_survives_a_role_that_lags_far_behind(starved):
    rng = random.Random(sum(map(ord, starved)))
    for n_iter in (1, 3, 4, 9, 18):
        backward_pipe(n_iter, rng, 5, starved=starved)

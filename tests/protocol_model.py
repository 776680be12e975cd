"""Discrete-event model of the mbarrier protocol of the key-loop tcgen05 kernels
(llsa_b200/csrc/attn_pooled_loop_tc.cu, attn_pooled_bwd_loop_tc.cu, attn_pooled_dkv_loop_tc.cu) of the
single-shot pooled forward and backward (attn_pooled_tc.cu, attn_pooled_bwd_tc.cu) and of the coarse selection (topk_tc.cu).

Test infrastructure: nothing in the package imports it.  Every role of a CTA
(the two TMA producers, the warps that issue MMAs, the softmax warps, the
four epilogue warps) is a Python generator that waits on barriers, spends random
time and arrives, exactly in the order the kernel's role does.  The model keeps the hardware's semantics where
they matter for correctness:

* a barrier has an arrival count and a phase; a wait names a PARITY and passes
  when the barrier's current (incomplete) phase has the other parity.  A wait
  for "completion number u" therefore also passes when completion u - 1 has
  not happened yet -- the case a protocol must exclude by construction;
* `tcgen05.commit` arrives when the MMAs the committing thread issued before
  it have completed; MMAs of all threads share one in-order pipe;
* a TMA load arrives on its barrier after a random latency.

On top of that the model tracks who owns each tensor-memory buffer and each
operand ring stage and asserts at every read and overwrite, so that a protocol
error shows as a failed assertion or as a deadlock (roles left waiting with no
event pending), not as a wrong number.
"""
import heapq
import random


class Barrier:
    def __init__(self, name, count):
        self.name, self.count, self.pending, self.phase = name, count, count, 0

    def parity(self):                     # parity of the current, incomplete phase
        return self.phase & 1

    def arrive(self, sim):
        self.pending -= 1
        assert self.pending >= 0, self.name
        if self.pending == 0:
            self.phase += 1
            self.pending = self.count
            sim.wake(self)


class Sim:
    def __init__(self, seed):
        self.t, self.queue, self.serial = 0, [], 0
        self.rng = random.Random(seed)
        self.waiting = []                 # (role, [(barrier, parity)])
        self.roles = {}
        self.pipe_free = 0                # the tensor pipe executes in issue order
        self.last_mma_done = {}           # per issuing thread

    def at(self, t, fn):
        self.serial += 1
        heapq.heappush(self.queue, (t, self.serial, fn))

    def spawn(self, name, gen):
        self.roles[name] = gen
        self.at(0, lambda: self.step(name))

    def step(self, name):
        gen = self.roles.get(name)
        if gen is None:
            return
        try:
            op = next(gen)
        except StopIteration:
            del self.roles[name]
            return
        if op[0] == "delay":
            self.at(self.t + op[1], lambda: self.step(name))
        else:                             # ("wait", barrier, parity[, barrier, parity ...]): all of them in one look
            conds = list(zip(op[1::2], op[2::2]))
            if all(b.parity() != par for b, par in conds):
                self.at(self.t + self.rng.randint(20, 120), lambda: self.step(name))
            else:
                self.waiting.append((name, conds))

    def wake(self, bar):
        still = []
        for name, conds in self.waiting:
            if any(b is bar for b, _ in conds) and all(b.parity() != par for b, par in conds):
                self.at(self.t + self.rng.randint(20, 150), (lambda nm: (lambda: self.step(nm)))(name))
            else:
                still.append((name, conds))
        self.waiting = still

    def run(self):
        while self.queue:
            self.t, _, fn = heapq.heappop(self.queue)
            fn()
        return "deadlock" if self.roles else "ok"

    def mma(self, thread, cycles):        # -> (start, done) on the shared pipe
        start = max(self.pipe_free, self.t)
        self.pipe_free = start + cycles
        self.last_mma_done[thread] = self.pipe_free
        return start, self.pipe_free

    def commit(self, thread, bar):
        done = max(self.last_mma_done.get(thread, 0), self.t) + self.rng.randint(20, 100)
        self.at(done, lambda: bar.arrive(self))

    def tma(self, bar, fn=None):
        def land():
            if fn:
                fn()
            bar.arrive(self)
        self.at(self.t + self.rng.randint(500, 1500), land)

    def r(self, a, b):
        return self.rng.randint(a, b)


class Resource:
    """A buffer with one content tag; reads must see the expected tag, and an overwrite must come after the last read
    (an MMA reads until it completes) has ended."""
    def __init__(self, name):
        self.name, self.tag, self.busy_until = name, None, 0

    def read(self, sim, tag, until=None):
        assert self.tag == tag, ("%s read" % self.name, self.tag, tag)
        self.busy_until = max(self.busy_until, sim.t if until is None else until)

    def write(self, sim, tag, at=None):
        assert sim.t >= self.busy_until, ("%s overwritten while it is read" % self.name, self.tag, tag, sim.t, self.busy_until)
        if at is None:
            self.tag = tag
        else:
            self.tag = ("in flight", tag)
            sim.at(at, (lambda: setattr(self, "tag", tag)))


def _bars(name, n, count):
    return [Barrier("%s%d" % (name, i), count) for i in range(n)]


def key_major_kernel(seed, units, score_threads=1, score_barriers=None, stages=8, buffers=None, full_count=2, dp_count=4,
                     dp_back_first=False):
    """attn_dkv_pooled_loop_tc_kernel.  `units`: job counts of the units of one CTA's piece: long (head, chunk) units, or, gathered, units of four
    jobs and fewer.  Four S^T buffers, which P^T and dS^T overwrite, one pair of accumulators, and two dP^T buffers, handed back as soon as their
    group has loaded them.  stages: of the Q / dO ring (8; gathered 4).  Two score threads share three S^T buffers.
    dp_count: warps whose arrivals hand a dP^T buffer back (4 = the kernel; fewer break the protocol on purpose), dp_back_first: a warp
    arrives before it has loaded its part (the same).
    score_threads: threads that issue S^T / dP^T (1 = the kernel; 2 = even and odd jobs on two threads).
    score_barriers: sdp_ready / buf_free barriers (None = one per buffer, the kernel; 6 = one per job number mod 6).
    full_count: producers a query stage waits for (2 = the kernel: Q, and dO with lse and delta; 1 breaks the protocol on purpose)."""
    sim = Sim(seed)
    accs = 1
    buffers = buffers or (4 if score_threads == 1 else 3)
    nb = score_barriers or buffers
    dp = [Resource("dP^T buffer %d" % i) for i in range(2)]
    dp_free = _bars("dp_free", 2, dp_count)
    kv_full, kv_empty = _bars("kv_full", 2, 1), _bars("kv_empty", 2, score_threads)
    q_full, q_empty = _bars("q_full", stages, full_count), _bars("q_empty", stages, 1)
    sdp, pds, free = _bars("sdp_ready", nb, 1), _bars("pds_ready", buffers, 4), _bars("buf_free", nb, 1)
    acc_ready, acc_free = _bars("acc_ready", accs, 1), _bars("acc_free", accs, 4)
    owner = [None] * buffers              # None: free; ("s", job): scores; ("p", job): probabilities
    keys = [Resource("key stage %d" % i) for i in range(2)]
    tiles = {n: [Resource("%s stage %d" % (n, i)) for i in range(stages)] for n in ("Q", "dO")}
    acc = [Resource("accumulator %d" % i) for i in range(accs)]

    def producer(which):
        job = 0
        for i, n in enumerate(units):
            if which == "Q":              # this producer also loads the unit's keys and values
                yield ("wait", kv_empty[i & 1], ((i >> 1) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                keys[i & 1].write(sim, i, at=land)
                sim.at(land, (lambda b=kv_full[i & 1]: b.arrive(sim)))
            for _ in range(n):
                st = job % stages
                yield ("wait", q_empty[st], ((job // stages) & 1) ^ 1)
                yield ("delay", sim.r(20, 80))
                land = sim.t + sim.r(500, 1500)
                tiles[which][st].write(sim, job, at=land)
                if which == "Q" or full_count == 2:
                    sim.at(land, (lambda b=q_full[st]: b.arrive(sim)))
                job += 1

    def score_issuer(mine):
        job, first = mine, 0
        for i, n in enumerate(units):
            yield ("wait", kv_full[i & 1], (i >> 1) & 1)
            while job < first + n:
                st, buf = job % stages, job % buffers
                wait = ["wait", q_full[st], (job // stages) & 1]
                if job >= buffers:
                    prev = job - buffers
                    wait += [free[prev % nb], (prev // nb) & 1]
                if job >= 2:
                    wait += [dp_free[job & 1], ((job >> 1) - 1) & 1]
                yield tuple(wait)
                if sim.rng.random() < 0.15:
                    yield ("delay", sim.r(500, 4000))          # one thread falls behind the other
                assert owner[buf] is None, ("scores written over a live buffer", buf, owner[buf], job)
                start, done = sim.mma(("score", mine), 384)
                keys[i & 1].read(sim, i, done)
                for t in tiles.values():
                    t[st].read(sim, job, done)
                sim.at(done, (lambda b=buf, j=job: owner.__setitem__(b, ("s", j))))
                dp[job & 1].write(sim, job, at=done)
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                sim.commit(("score", mine), sdp[job % nb])
                yield ("delay", sim.r(30, 80))
                job += score_threads
            first += n
            sim.commit(("score", mine), kv_empty[i & 1])
            yield ("delay", sim.r(30, 80))

    def out_issuer():
        job = 0
        for i, n in enumerate(units):
            for j in range(n):
                st, buf = job % stages, job % buffers
                wait = ["wait", pds[buf], (job // buffers) & 1]
                if j == 0 and i >= accs:
                    wait += [acc_free[i % accs], (i // accs - 1) & 1]
                yield tuple(wait)
                assert owner[buf] == ("p", job), ("dV / dK read", buf, owner[buf], job)
                start, done = sim.mma("out", 384)
                for t in tiles.values():
                    t[st].read(sim, job, done)
                if j == 0:
                    acc[i % accs].write(sim, i)
                sim.at(done, (lambda b=buf: owner.__setitem__(b, None)))
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                sim.commit("out", q_empty[st])
                sim.commit("out", free[job % nb])
                yield ("delay", sim.r(60, 160))
                job += 1
            sim.commit("out", acc_ready[i % accs])
            yield ("delay", sim.r(30, 80))

    def softmax(group, warp):
        for job in range(group, sum(units), 2):
            buf = job % buffers
            yield ("wait", sdp[job % nb], (job // nb) & 1)
            assert owner[buf] is not None and owner[buf][1] == job, ("softmax read", buf, owner[buf], job)
            if dp_back_first:
                dp_free[job & 1].arrive(sim)
            yield ("delay", sim.r(100, 400))
            dp[job & 1].read(sim, job)
            if not dp_back_first:
                dp_free[job & 1].arrive(sim)
            yield ("delay", sim.r(500, 1200))
            if warp == 0:
                owner[buf] = ("p", job)
            pds[buf].arrive(sim)

    def epilogue(warp):
        for i in range(len(units)):
            a = i % accs
            yield ("wait", acc_ready[a], (i // accs) & 1)
            acc[a].read(sim, i)
            yield ("delay", sim.r(200, 1500))
            acc[a].read(sim, i)
            acc_free[a].arrive(sim)

    for which in ("Q", "dO"):
        sim.spawn("producer " + which, producer(which))
    for t in range(score_threads):
        sim.spawn("score%d" % t, score_issuer(t))
    sim.spawn("out", out_issuer())
    for w in range(4):
        for g in range(2):
            sim.spawn("softmax%d%d" % (g, w), softmax(g, w))
        sim.spawn("epilogue%d" % w, epilogue(w))
    return sim.run()


def query_major_kernel(seed, tiles, jobs, score_threads=1, score_barriers=None, stages=8, buffers=None, free_count=4, dp_count=4, dp_back_first=False):
    """attn_dq_pooled_loop_tc_kernel: `tiles` query tiles of `jobs` key chunks; Q / dO in two stages, K and V chunks (two
    producers) in one ring of pairs, S into four buffers (three with two score threads), which dS overwrites, dP into two, handed back as soon
    as their group has loaded them, dQ of a tile into one of two accumulators, read by epilogue warps.
    free_count: epilogue warps an accumulator waits for (4 = the kernel; 1 breaks the protocol on purpose); dp_count, dp_back_first: as in
    key_major_kernel."""
    sim = Sim(seed)
    buffers = buffers or (4 if score_threads == 1 else 3)
    nb = score_barriers or buffers
    dp = [Resource("dP buffer %d" % i) for i in range(2)]
    dp_free = _bars("dp_free", 2, dp_count)
    q_full, q_empty = _bars("q_full", 2, 1), _bars("q_empty", 2, score_threads)
    kv_full, kv_empty = _bars("kv_full", stages, 2), _bars("kv_empty", stages, 1)
    sdp, ds, free = _bars("sdp_ready", nb, 1), _bars("ds_ready", buffers, 4), _bars("buf_free", nb, 1)
    dq_ready, dq_free = _bars("dq_ready", 2, 1), _bars("dq_free", 2, free_count)
    owner = [None] * buffers
    ring = {n: [Resource("%s stage %d" % (n, i)) for i in range(stages)] for n in ("K", "V")}
    q_tile = [Resource("Q / dO stage %d" % i) for i in range(2)]
    acc = [Resource("dQ accumulator %d" % i) for i in range(2)]

    def producer(which):
        job = 0
        for i in range(tiles):
            if which == "K":              # this producer also loads Q and dO
                yield ("wait", q_empty[i & 1], ((i >> 1) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                q_tile[i & 1].write(sim, i, at=land)
                sim.at(land, (lambda b=q_full[i & 1]: b.arrive(sim)))
            for _ in range(jobs):
                st = job % stages
                yield ("wait", kv_empty[st], ((job // stages) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                ring[which][st].write(sim, job, at=land)
                sim.at(land, (lambda b=kv_full[st]: b.arrive(sim)))
                job += 1

    def score_issuer(mine):
        job = mine
        for i in range(tiles):
            yield ("wait", q_full[i & 1], (i >> 1) & 1)
            while job < (i + 1) * jobs:
                st, buf = job % stages, job % buffers
                wait = ["wait", kv_full[st], (job // stages) & 1]
                if job >= buffers:
                    prev = job - buffers
                    wait += [free[prev % nb], (prev // nb) & 1]
                if job >= 2:
                    wait += [dp_free[job & 1], ((job >> 1) - 1) & 1]
                yield tuple(wait)
                if sim.rng.random() < 0.15:
                    yield ("delay", sim.r(500, 4000))
                assert owner[buf] is None, ("scores written over a live buffer", buf, owner[buf], job)
                start, done = sim.mma(("score", mine), 384)
                q_tile[i & 1].read(sim, i, done)
                for r in ring.values():
                    r[st].read(sim, job, done)
                sim.at(done, (lambda b=buf, j=job: owner.__setitem__(b, ("s", j))))
                dp[job & 1].write(sim, job, at=done)
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                sim.commit(("score", mine), sdp[job % nb])
                yield ("delay", sim.r(30, 80))
                job += score_threads
            sim.commit(("score", mine), q_empty[i & 1])
            yield ("delay", sim.r(30, 80))

    def dq_issuer():
        job = 0
        for i in range(tiles):
            for j in range(jobs):
                st, buf = job % stages, job % buffers
                wait = ["wait", ds[buf], (job // buffers) & 1]
                if j == 0 and i > 1:
                    wait += [dq_free[i & 1], ((i - 2) >> 1) & 1]
                yield tuple(wait)
                assert owner[buf] == ("p", job), ("dQ read", buf, owner[buf], job)
                start, done = sim.mma("dq", 192)
                ring["K"][st].read(sim, job, done)
                if j == 0:
                    acc[i & 1].write(sim, i)
                sim.at(done, (lambda b=buf: owner.__setitem__(b, None)))
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                sim.commit("dq", kv_empty[st])
                sim.commit("dq", free[job % nb])
                yield ("delay", sim.r(60, 160))
                job += 1
            sim.commit("dq", dq_ready[i & 1])
            yield ("delay", sim.r(30, 80))

    def softmax(group, warp):
        for job in range(group, tiles * jobs, 2):
            buf = job % buffers
            yield ("wait", sdp[job % nb], (job // nb) & 1)
            assert owner[buf] is not None and owner[buf][1] == job, ("softmax read", buf, owner[buf], job)
            if dp_back_first:
                dp_free[job & 1].arrive(sim)
            yield ("delay", sim.r(100, 400))
            dp[job & 1].read(sim, job)
            if not dp_back_first:
                dp_free[job & 1].arrive(sim)
            yield ("delay", sim.r(400, 1000))
            if warp == 0:
                owner[buf] = ("p", job)
            ds[buf].arrive(sim)

    def epilogue(warp):
        for i in range(tiles):
            yield ("wait", dq_ready[i & 1], (i >> 1) & 1)
            acc[i & 1].read(sim, i)
            yield ("delay", sim.r(200, 3000))
            acc[i & 1].read(sim, i)
            if warp < free_count:
                dq_free[i & 1].arrive(sim)

    for which in ("K", "V"):
        sim.spawn("producer " + which, producer(which))
    for t in range(score_threads):
        sim.spawn("score%d" % t, score_issuer(t))
    sim.spawn("dq", dq_issuer())
    for w in range(4):
        for g in range(2):
            sim.spawn("softmax%d%d" % (g, w), softmax(g, w))
        sim.spawn("epilogue%d" % w, epilogue(w))
    return sim.run()


def forward_kernel(seed, tiles, chunks, passes, k_stages=4, v_stages=4, buffers=3, groups=3, second_round=False, softmax_waits_for_sums=True):
    """attn_fwd_pooled_loop_tc_kernel: `tiles` query tiles of `chunks` key chunks; one pass (jobs = chunks, every job
    feeds P.V) or two (jobs = 2 * chunks: row maxima first, then the exponentials; the groups exchange their maxima
    once per tile, a group without a second-pass job at its end).  Producers of keys (with Q) and of values; one warp issues S, one P.V
    and hands every job's buffer back; softmax group g of `groups` (three, or two for short lists) takes the jobs whose CTA-wide number is g mod
    groups (of three always the same buffer; a tile's first job goes round the groups) and leaves its row sums to four epilogue warps, as O in
    one of two accumulators.
    second_round: the CTA has marked a row and goes over its tiles again with two passes, on barriers of its own, behind a CTA-wide
    synchronisation.  softmax_waits_for_sums=False breaks the protocol on purpose (row sums overwritten before they are read)."""
    sim = Sim(seed)
    owner = [None] * buffers
    k_ring = [Resource("K stage %d" % i) for i in range(k_stages)]
    v_ring = [Resource("V stage %d" % i) for i in range(v_stages)]
    q_tile = [Resource("Q stage %d" % i) for i in range(2)]
    acc = [Resource("O accumulator %d" % i) for i in range(2)]
    sums = [[Resource("row sums %d of group %d" % (i, g)) for g in range(groups)] for i in range(2)]
    maxima = [[Resource("row maxima %d of group %d" % (i, g)) for g in range(groups)] for i in range(2)]
    n_roles = 2 + 2 + 4 * groups + 4
    sync = Barrier("__syncthreads", n_roles)

    class Round:
        def __init__(self, number, passes):
            self.number, self.passes = number, passes
            self.jobs, self.first_p2 = passes * chunks, (passes - 1) * chunks
            self.q_full, self.q_empty = _bars("q_full", 2, 1), _bars("q_empty", 2, 1)
            self.k_full, self.k_empty = _bars("k_full", k_stages, 1), _bars("k_empty", k_stages, 1)
            self.v_full, self.v_empty = _bars("v_full", v_stages, 1), _bars("v_empty", v_stages, 1)
            self.s_ready, self.wg_done, self.free = _bars("s_ready", buffers, 1), _bars("wg_done", buffers, 4), _bars("buf_free", buffers, 1)
            self.o_ready, self.o_free, self.sum_ready = _bars("o_ready", 2, 1), _bars("o_free", 2, 4), _bars("sum_ready", 2, 4 * groups)
            self.xchg = Barrier("xchg", 4 * groups)

    rounds = [Round(0, passes)] + ([Round(1, 2)] if second_round else [])

    def producer(x, which):
        stages, full, empty, ring = ((k_stages, x.k_full, x.k_empty, k_ring) if which == "K" else (v_stages, x.v_full, x.v_empty, v_ring))
        n = 0
        for i in range(tiles):
            if which == "K":
                yield ("wait", x.q_empty[i & 1], ((i >> 1) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                q_tile[i & 1].write(sim, (x.number, i), at=land)
                sim.at(land, (lambda b=x.q_full[i & 1]: b.arrive(sim)))
            for _ in range(x.jobs if which == "K" else chunks):
                st = n % stages
                yield ("wait", empty[st], ((n // stages) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                ring[st].write(sim, (x.number, n), at=land)
                sim.at(land, (lambda b=full[st]: b.arrive(sim)))
                n += 1

    def s_issuer(x):
        n = 0
        for i in range(tiles):
            yield ("wait", x.q_full[i & 1], (i >> 1) & 1)
            for _ in range(x.jobs):
                buf, ks = n % buffers, n % k_stages
                wait = ["wait", x.k_full[ks], (n // k_stages) & 1]
                if n >= buffers:
                    wait += [x.free[buf], ((n // buffers) & 1) ^ 1]
                yield tuple(wait)
                assert owner[buf] is None, ("scores written over a live buffer", buf, owner[buf], n)
                start, done = sim.mma("s", 256)
                q_tile[i & 1].read(sim, (x.number, i), done)
                k_ring[ks].read(sim, (x.number, n), done)
                sim.at(done, (lambda b=buf, j=n: owner.__setitem__(b, ("s", j))))
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                sim.commit("s", x.s_ready[buf])
                sim.commit("s", x.k_empty[ks])
                yield ("delay", sim.r(30, 80))
                n += 1
            sim.commit("s", x.q_empty[i & 1])
            yield ("delay", sim.r(30, 80))

    def pv_issuer(x):
        n = vjob = 0
        for i in range(tiles):
            for j in range(x.jobs):
                buf, vs, pv = n % buffers, vjob % v_stages, j >= x.first_p2
                wait = ["wait", x.wg_done[buf], (n // buffers) & 1]
                if pv:
                    wait += [x.v_full[vs], (vjob // v_stages) & 1]
                    if j == x.first_p2 and i > 1:
                        wait += [x.o_free[i & 1], ((i - 2) >> 1) & 1]
                yield tuple(wait)
                if pv:
                    assert owner[buf] == ("p", n), ("P.V read", buf, owner[buf], n)
                    start, done = sim.mma("pv", 384)
                    v_ring[vs].read(sim, (x.number, vjob), done)
                    if j == x.first_p2:
                        acc[i & 1].write(sim, (x.number, i))
                    sim.at(done, (lambda b=buf: owner.__setitem__(b, None)))
                    yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                    sim.commit("pv", x.v_empty[vs])
                    vjob += 1
                else:
                    assert owner[buf] == ("m", n), ("first-pass buffer handed back early", buf, owner[buf], n)
                    owner[buf] = None
                sim.commit("pv", x.free[buf])
                yield ("delay", sim.r(30, 80))
                n += 1
            sim.commit("pv", x.o_ready[i & 1])
            yield ("delay", sim.r(30, 80))

    def softmax(x, group, warp):
        n = group                         # this group's next job, numbered over the CTA

        def exchange(i):
            slot = maxima[i & 1][group]
            if warp == 0:
                slot.write(sim, (x.number, i))
            x.xchg.arrive(sim)
            yield ("wait", x.xchg, i & 1)
            for g in range(groups):
                maxima[i & 1][g].read(sim, (x.number, i))

        for i in range(tiles):
            j = (group - i * x.jobs) % groups
            assert j >= x.jobs or i * x.jobs + j == n, ("job numbering", i, j, n)
            exchanged = x.passes == 1
            while j < x.jobs:
                buf = n % buffers
                if j >= x.first_p2 and not exchanged:
                    exchanged = True
                    yield from exchange(i)
                yield ("wait", x.s_ready[buf], (n // buffers) & 1)
                assert owner[buf] is not None and owner[buf][1] == n, ("softmax read", buf, owner[buf], n)
                yield ("delay", sim.r(400, 1400))
                if warp == 0:
                    owner[buf] = ("p" if j >= x.first_p2 else "m", n)
                x.wg_done[buf].arrive(sim)
                n += groups
                j += groups
            if not exchanged:
                yield from exchange(i)
            if i > 1 and softmax_waits_for_sums:
                yield ("wait", x.o_free[i & 1], ((i - 2) >> 1) & 1)
            if warp == 0:
                sums[i & 1][group].write(sim, (x.number, i))
            x.sum_ready[i & 1].arrive(sim)

    def epilogue(x, warp):
        for i in range(tiles):
            yield ("wait", x.sum_ready[i & 1], (i >> 1) & 1)
            yield ("wait", x.o_ready[i & 1], (i >> 1) & 1)
            for _ in range(2):
                for r in (acc[i & 1], *sums[i & 1]):
                    r.read(sim, (x.number, i))
                yield ("delay", sim.r(100, 2500))
            acc[i & 1].read(sim, (x.number, i))
            x.o_free[i & 1].arrive(sim)

    def all_rounds(role, *args):
        for x in rounds:
            yield from role(x, *args)
            sync.arrive(sim)
            yield ("wait", sync, x.number & 1)

    for which in ("K", "V"):
        sim.spawn("producer " + which, all_rounds(producer, which))
    sim.spawn("s", all_rounds(s_issuer))
    sim.spawn("pv", all_rounds(pv_issuer))
    for w in range(4):
        for g in range(groups):
            sim.spawn("softmax%d%d" % (g, w), all_rounds(softmax, g, w))
        sim.spawn("epilogue%d" % w, all_rounds(epilogue, w))
    return sim.run()


def single_shot_backward_kernel(seed, t_begin, n_tiles, tiles_per_head, mma_done_count=2, softmax_waits_for_products=True):
    """attn_bwd_pooled_tc_kernel: tiles [t_begin, t_begin + n_tiles) of one CTA; a parent is two tiles (even, odd), a head is
    tiles_per_head tiles (even).  Two MMA-issuing threads: A = S, dP, dQ; B = the three transposed products.
    The last two arguments break the protocol on purpose (tests of the model itself): mma_done counting only thread A's
    commit, and softmax warps that overwrite P / dS without waiting for the previous tile's products."""
    sim = Sim(seed)
    full = [Barrier("full%d" % i, 1) for i in range(2)]
    mma_done = [Barrier("mma_done%d" % i, mma_done_count) for i in range(2)]
    v_free = [Barrier("v_free%d" % i, 1) for i in range(2)]
    s_ready, dp_ready, out_ready = Barrier("s_ready", 1), Barrier("dp_ready", 1), Barrier("out_ready", 2)
    s_consumed, pds_ready = Barrier("s_consumed", 12), Barrier("pds_ready", 12)
    dq_free, acc_free = Barrier("dq_free", 4), Barrier("acc_free", 4)
    stage = [Resource("Q/dO stage %d" % i) for i in range(2)]
    k1 = [Resource("K1 buffer %d" % i) for i in range(2)]
    v1, kv2 = Resource("V1"), Resource("K2/V2")
    scores, pds, dq = Resource("S/dP columns"), Resource("P/dS tiles"), Resource("dQ columns")
    acc1, acc2 = Resource("level-1 accumulators"), Resource("level-2 accumulators")
    tile_of = lambda i: t_begin + i
    parent_of = lambda i: tile_of(i) >> 1
    head_of = lambda i: tile_of(i) // tiles_per_head

    def producer():
        for i in range(n_tiles):
            s, tile = i & 1, tile_of(i)
            new_parent = i == 0 or tile % 2 == 0
            new_head = i == 0 or tile % tiles_per_head == 0
            if i >= 2:
                yield ("wait", mma_done[s], ((i - 2) >> 1) & 1)
            if i >= 1 and new_head:
                yield ("wait", mma_done[(i - 1) & 1], ((i - 1) >> 1) & 1)
            land = sim.t + sim.r(500, 1500)
            stage[s].write(sim, tile, at=land)
            if new_head:
                kv2.write(sim, head_of(i), at=land)
            if new_parent:
                k1[parent_of(i) & 1].write(sim, parent_of(i), at=land)
                if i >= 1:
                    yield ("wait", v_free[(i - 1) & 1], ((i - 1) >> 1) & 1)
                land = max(land, sim.t + sim.r(500, 1500))
                v1.write(sim, parent_of(i), at=land)
            sim.at(land, (lambda b=full[s]: b.arrive(sim)))
            yield ("delay", sim.r(20, 80))

    def issuer_a():
        def issue_s(i):
            s = i & 1
            yield ("wait", full[s], (i >> 1) & 1)
            start, done = sim.mma("A", 384)
            stage[s].read(sim, tile_of(i), done)
            k1[parent_of(i) & 1].read(sim, parent_of(i), done)
            kv2.read(sim, head_of(i), done)
            scores.write(sim, ("S", i), at=done)
            yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
            sim.commit("A", s_ready)

        if n_tiles > 0:
            yield from issue_s(0)
        for i in range(n_tiles):
            s, tile = i & 1, tile_of(i)
            yield ("wait", s_consumed, i & 1)
            start, done = sim.mma("A", 384)
            stage[s].read(sim, tile, done)
            v1.read(sim, parent_of(i), done)
            kv2.read(sim, head_of(i), done)
            scores.write(sim, ("dP", i), at=done)
            yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
            sim.commit("A", dp_ready)
            sim.commit("A", v_free[s])
            yield ("wait", pds_ready, i & 1)
            next_early = i + 1 < n_tiles and (tile + 1) % tiles_per_head != 0
            if next_early:
                yield from issue_s(i + 1)
            if i > 0:
                yield ("wait", dq_free, (i - 1) & 1)
            start, done = sim.mma("A", 576)
            pds.read(sim, i, done)
            k1[parent_of(i) & 1].read(sim, parent_of(i), done)
            kv2.read(sim, head_of(i), done)
            dq.write(sim, i, at=done)
            yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
            sim.commit("A", out_ready)
            sim.commit("A", mma_done[s])
            if not next_early and i + 1 < n_tiles:
                yield from issue_s(i + 1)

    def issuer_b():
        parents_done = 0
        for i in range(n_tiles):
            s, tile = i & 1, tile_of(i)
            yield ("wait", pds_ready, i & 1)
            fresh1 = not (i > 0 and tile % 2 == 1)
            fresh2 = not (i > 0 and tile % tiles_per_head != 0)
            if fresh1 and parents_done > 0:
                yield ("wait", acc_free, (parents_done - 1) & 1)
            start, done = sim.mma("B", 1280)
            pds.read(sim, i, done)
            stage[s].read(sim, tile, done)
            if fresh1:
                acc1.write(sim, parent_of(i))
            else:
                acc1.read(sim, parent_of(i))
            if fresh2:
                acc2.write(sim, head_of(i))
            else:
                acc2.read(sim, head_of(i))
            acc1.busy_until = max(acc1.busy_until, 0)
            yield ("delay", max(0, start - sim.t) + sim.r(50, 300))
            sim.commit("B", out_ready)
            if mma_done_count == 2:
                sim.commit("B", mma_done[s])
            if tile % 2 == 1 or i == n_tiles - 1:
                parents_done += 1

    def drain(warp):
        for i in range(n_tiles):
            tile = tile_of(i)
            parent_end = tile % 2 == 1 or i == n_tiles - 1
            yield ("wait", out_ready, i & 1)
            dq.read(sim, i)
            yield ("delay", sim.r(150, 400))
            dq.busy_until = max(dq.busy_until, sim.t)
            dq_free.arrive(sim)
            if not parent_end:
                continue
            acc1.read(sim, parent_of(i))
            if i == n_tiles - 1 or (tile + 1) % tiles_per_head == 0:
                acc2.read(sim, head_of(i))
            yield ("delay", sim.r(300, 900))
            acc1.busy_until = max(acc1.busy_until, sim.t)
            acc2.busy_until = max(acc2.busy_until, sim.t)
            acc_free.arrive(sim)

    def softmax(warp):
        for i in range(n_tiles):
            yield ("wait", s_ready, i & 1)
            scores.read(sim, ("S", i))
            yield ("delay", sim.r(200, 500))
            scores.busy_until = max(scores.busy_until, sim.t)
            s_consumed.arrive(sim)
            if i > 0 and softmax_waits_for_products:
                yield ("wait", out_ready, (i - 1) & 1)
            if warp == 0:
                pds.write(sim, ("being written", i))
            yield ("delay", sim.r(100, 300))
            yield ("wait", dp_ready, i & 1)
            scores.read(sim, ("dP", i))
            yield ("delay", sim.r(300, 700))
            scores.busy_until = max(scores.busy_until, sim.t)
            if warp == 0:
                pds.tag = i
            pds_ready.arrive(sim)

    sim.spawn("producer", producer())
    sim.spawn("A", issuer_a())
    sim.spawn("B", issuer_b())
    for w in range(4):
        sim.spawn("drain%d" % w, drain(w))
    for w in range(12):
        sim.spawn("softmax%d" % w, softmax(w))
    return sim.run()

def single_shot_forward_kernel(seed, tiles, head=True, sums_wait_for_epilogue=True, products_wait_for_epilogue=True, o_ring=3):
    """attn_fwd_pooled_tc_kernel: `tiles` query tiles of one CTA, two score buffers (P over S, O behind them).  Two producers (Q and keys, three
    stages; values, two), one warp issues S, one O = P.V, two softmax groups on alternate tiles, four epilogue warps, each with its own rows of o:
    loaded a tile ahead into a ring of three, merged in place and stored from there.
    head: P of all but the last 64 keys is handed over first (more than 64 keys).  The last three arguments break the protocol on purpose:
    maxima and sums written before the tile before last's have been read, O written before it has been read, an o ring that is too short for
    the store that may still read it."""
    sim = Sim(seed)
    key_stages, value_stages = 3, 2
    owner = [None, None]
    keys = [Resource("Q / key stage %d" % i) for i in range(key_stages)]
    values = [Resource("value stage %d" % i) for i in range(value_stages)]
    acc = [Resource("O of buffer %d" % i) for i in range(2)]
    stats = [Resource("maxima and sums %d" % i) for i in range(2)]
    full_k, empty_k = _bars("full_k", key_stages, 1), _bars("empty_k", key_stages, 1)
    full_v, empty_v = _bars("full_v", value_stages, 1), _bars("empty_v", value_stages, 1)
    s_ready, p_head, p_ready = _bars("s_ready", 2, 1), _bars("p_head", 2, 4), _bars("p_ready", 2, 4)
    buf_free, o_ready, o_free = _bars("buf_free", 2, 1), _bars("o_ready", 2, 1), _bars("o_free", 2, 4)

    def producer(ring, full, empty, stages):
        for i in range(tiles):
            st = i % stages
            yield ("wait", empty[st], ((i // stages) & 1) ^ 1)
            land = sim.t + sim.r(500, 1500)
            ring[st].write(sim, i, at=land)
            sim.at(land, (lambda b=full[st]: b.arrive(sim)))

    def s_issuer():
        for i in range(tiles):
            st, b = i % key_stages, i & 1
            wait = ["wait", full_k[st], (i // key_stages) & 1]
            if i >= 2:
                wait += [buf_free[b], ((i >> 1) - 1) & 1]
            yield tuple(wait)
            assert owner[b] is None, ("scores written over a live buffer", b, owner[b], i)
            start, done = sim.mma("s", 384)
            keys[st].read(sim, i, done)
            sim.at(done, (lambda b=b, i=i: owner.__setitem__(b, ("s", i))))
            yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
            sim.commit("s", s_ready[b])
            sim.commit("s", empty_k[st])
            yield ("delay", sim.r(30, 80))

    def o_issuer():
        for i in range(tiles):
            st, b, par = i % value_stages, i & 1, (i >> 1) & 1
            wait = ["wait", full_v[st], (i // value_stages) & 1, (p_head if head else p_ready)[b], par]
            if i >= 2 and products_wait_for_epilogue:
                wait += [o_free[b], par ^ 1]
            yield tuple(wait)
            acc[b].write(sim, i)
            if head:
                assert owner[b] in (("h", i), ("p", i)), ("first part of P.V read", b, owner[b], i)
                start, done = sim.mma("o", 384)
                values[st].read(sim, i, done)
                yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                yield ("wait", p_ready[b], par)
            assert owner[b] == ("p", i), ("P.V read", b, owner[b], i)
            start, done = sim.mma("o", 192)
            values[st].read(sim, i, done)
            sim.at(done, (lambda b=b: owner.__setitem__(b, None)))
            yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
            for bar in (o_ready[b], empty_v[st], buf_free[b]):
                sim.commit("o", bar)
            yield ("delay", sim.r(30, 80))

    def softmax(group, warp):
        for i in range(group, tiles, 2):
            par = (i >> 1) & 1
            yield ("wait", s_ready[group], par)
            assert owner[group] is not None and owner[group][1] == i, ("softmax read", group, owner[group], i)
            yield ("delay", sim.r(600, 2000))
            if head:
                if warp == 0:
                    owner[group] = ("h", i)
                p_head[group].arrive(sim)
                yield ("delay", sim.r(200, 600))
            if i >= 2 and sums_wait_for_epilogue:
                yield ("wait", o_free[group], par ^ 1)
            if warp == 0:
                stats[group].write(sim, ("being written", i))
                owner[group] = ("p", i)
            yield ("delay", sim.r(5, 30))
            if warp == 0:
                stats[group].tag = i
            p_ready[group].arrive(sim)

    def epilogue(warp):
        ring = [Resource("o stage %d of warp %d" % (i, warp)) for i in range(o_ring)]
        full = _bars("out_full", o_ring, 1)
        stored = []                       # when the stores issued so far have read their stage

        def request(i):
            land = sim.t + sim.r(500, 1500)
            ring[i % o_ring].write(sim, i, at=land)
            sim.at(land, (lambda b=full[i % o_ring]: b.arrive(sim)))

        if tiles:
            request(0)
        for i in range(tiles):
            b, par = i & 1, (i >> 1) & 1
            if i + 1 < tiles:
                if len(stored) >= 2:      # all but the newest store have read their stage
                    yield ("delay", max(0, stored[-2] - sim.t))
                request(i + 1)
            yield ("wait", full[i % o_ring], (i // o_ring) & 1)
            yield ("wait", p_ready[b], par)
            yield ("wait", o_ready[b], par)
            for _ in range(2):
                for r in (acc[b], stats[b]):
                    r.read(sim, i)
                yield ("delay", sim.r(100, 2500))
            acc[b].read(sim, i)
            stats[b].read(sim, i)
            o_free[b].arrive(sim)
            yield ("delay", sim.r(50, 300))
            at = max([sim.t] + stored[-1:]) + sim.r(100, 3000)      # stores read in order
            ring[i % o_ring].read(sim, i, at)
            stored.append(at)

    sim.spawn("producer K", producer(keys, full_k, empty_k, key_stages))
    sim.spawn("producer V", producer(values, full_v, empty_v, value_stages))
    sim.spawn("s", s_issuer())
    sim.spawn("o", o_issuer())
    for w in range(4):
        for g in range(2):
            sim.spawn("softmax%d%d" % (g, w), softmax(g, w))
        sim.spawn("epilogue%d" % w, epilogue(w))
    return sim.run()


def coarse_selection_kernel(seed, shares, free_count=4, groups_meet=True, lists_wait=True):
    """coarse_topk_tc_kernel: a cluster whose CTA k walks shares[k] key chunks twice (a job each time).  One producer (two key stages), one warp issues
    the products, half a job at a time, two groups of four warps on alternate jobs, each with a score buffer per half of its job.  The groups of a CTA share
    the maxima of the first pass, the CTAs the bounds, then (pass 2 sets scores aside where the maxima were) the groups and in the end the CTAs
    their lists.
    free_count: warps whose arrivals hand a score buffer back (4 = the kernel); groups_meet=False: maxima read without the meeting that
    says they are written; lists_wait=False: a CTA leaves without waiting for the ones that read its lists.  Each breaks the protocol on purpose."""
    sim = Sim(seed)
    meet_count = 10 * len(shares)         # every warp of the cluster
    meet = [Barrier("cluster meeting %d" % i, meet_count) for i in range(3)]
    bound = [Resource("bound of CTA %d" % k) for k in range(len(shares))]
    lists = [Resource("lists of CTA %d" % k) for k in range(len(shares))]

    def cta(k, chunks):
        jobs = 2 * chunks
        stage = [Resource("key stage %d of CTA %d" % (i, k)) for i in range(2)]
        owner = {}
        place = [Resource("maxima / slots of group %d, CTA %d" % (g, k)) for g in range(2)]
        k_full, k_empty = _bars("k_full", 2, 1), _bars("k_empty", 2, 1)
        s_ready, s_free = _bars("s_ready", 4, 1), _bars("s_free", 4, free_count)
        pair = [Barrier("group_sync %d" % i, 8) for i in range(3)]
        sync = Barrier("__syncthreads", 10)

        def end(warp):
            sync.arrive(sim)
            yield ("wait", sync, 0)
            if warp == 0:
                lists[k].tag = "lists"
            meet[1].arrive(sim)
            yield ("wait", meet[1], 0)
            if warp < 4:
                for o in range(len(shares)):
                    lists[o].read(sim, "lists")
                yield ("delay", sim.r(50, 800))
                for o in range(len(shares)):
                    lists[o].read(sim, "lists")
            meet[2].arrive(sim)
            if lists_wait:
                yield ("wait", meet[2], 0)
            if warp == 0:
                lists[k].write(sim, "gone with the CTA")

        def producer():
            meet[0].arrive(sim)
            for j in range(jobs):
                yield ("wait", k_empty[j & 1], ((j >> 1) & 1) ^ 1)
                land = sim.t + sim.r(500, 1500)
                stage[j & 1].write(sim, j, at=land)
                sim.at(land, (lambda b=k_full[j & 1]: b.arrive(sim)))
            yield ("wait", meet[0], 0)
            yield from end(8)

        def issuer():
            meet[0].arrive(sim)
            for j in range(jobs):
                for half in range(2):
                    buf = (j & 1) * 2 + half
                    wait = ["wait", k_full[j & 1], (j >> 1) & 1]
                    if j >= 2:
                        wait += [s_free[buf], ((j >> 1) - 1) & 1]
                    yield tuple(wait)
                    assert owner.get(buf) is None, ("scores written over a live buffer", buf, owner[buf], j)
                    start, done = sim.mma(("s", k), 192)
                    stage[j & 1].read(sim, j, done)
                    owner[buf] = ("in flight", j)
                    sim.at(done, (lambda b=buf, j=j: owner.__setitem__(b, (j, 4))))
                    yield ("delay", max(0, start - sim.t) + sim.r(50, 200))
                    sim.commit(("s", k), s_ready[buf])
                sim.commit(("s", k), k_empty[j & 1])
                yield ("delay", sim.r(30, 80))
            yield ("wait", meet[0], 0)
            yield from end(9)

        def group(g, warp):
            def look(j, first):
                for half in range(2):
                    buf = g * 2 + half
                    yield ("wait", s_ready[buf], (j >> 1) & 1)
                    assert owner[buf] is not None and owner[buf][0] == j, ("scores read", buf, owner[buf], j)
                    yield ("delay", sim.r(100, 900))
                    assert owner[buf] is not None and owner[buf][0] == j, ("scores gone while they are read", buf, owner[buf], j)
                    left = owner[buf][1] - 1
                    owner[buf] = (j, left) if left else None
                    if warp < free_count:
                        s_free[buf].arrive(sim)
                    if not first and sim.rng.random() < 0.3:
                        yield ("delay", sim.r(200, 3000))

            for j in range(g, chunks, 2):
                yield from look(j, True)
            if warp == 0:
                place[g].tag = "maxima"
            pair[0].arrive(sim)
            if groups_meet:
                yield ("wait", pair[0], 0)
            for o in range(2):
                place[o].read(sim, "maxima", sim.t + 40)
            yield ("delay", sim.r(40, 200))
            if g == 0 and warp == 0:
                bound[k].tag = "bound"
            meet[0].arrive(sim)
            yield ("wait", meet[0], 0)
            for o in range(len(shares)):
                bound[o].read(sim, "bound")
            if warp == 0:
                place[g].write(sim, "slots")
            first2 = chunks + ((chunks & 1) ^ g)
            for j in range(first2, jobs, 2):
                yield from look(j, False)
            if warp == 0:                 # every warp has slots of its own; the model follows the first one's
                place[g].read(sim, "slots")
            pair[1].arrive(sim)
            yield ("wait", pair[1], 0)
            if g == 1 and warp == 0:
                place[1].write(sim, "list")
            pair[2].arrive(sim)
            yield ("wait", pair[2], 0)
            if g == 0:
                place[1].read(sim, "list")
            yield ("delay", sim.r(20, 100))
            yield from end(4 * g + warp)

        sim.spawn("producer %d" % k, producer())
        sim.spawn("s %d" % k, issuer())
        for w in range(4):
            for g in range(2):
                sim.spawn("group %d%d of %d" % (g, w, k), group(g, w))

    for k, chunks in enumerate(shares):
        cta(k, chunks)
    return sim.run()


def outcome(fn, *args, **kw):
    try:
        return fn(*args, **kw)
    except AssertionError as e:
        return "hazard: %s" % (e.args[0],)

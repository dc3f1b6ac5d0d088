"""The waits and arrivals of the tensor-core backward's warps, as a model that runs on the CPU.

Every role of the kernel (two soft-max warpgroups, two fold warpgroups, the issuing warps, the loader, the warps that form
R) is restated as the sequence of its barrier operations and of the buffers that it reads and writes; products and copies
finish later than they are issued, each issuer's in its order.  How many barriers stand behind a name (one, or two by step parity)
is read from the kernel's source.  A barrier is waited for by the parity of a phase, as the hardware does it, so one that is two
phases ahead of its waiter reads as not ready.

Checked: with any one role held back at any of its operations until nothing else can move, and for random orders, (1) every
role comes to its end, (2) every wait passes for a phase that is complete, (3) any two accesses to a buffer of which one writes
are ordered by barriers (vector clocks)."""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-3-way-attention_b200", "csrc",
                      "tritt_sm100_tdp_bwd.cu")
BATCH = SLOTS = 4


def _depths():
    """Barriers per name in the kernel's barrier block."""
    with open(SOURCE) as f:
        block = re.search(r"struct BwdBarriers \{(.*?)\n\};", f.read(), re.S).group(1)
    depths = {}
    for line in re.findall(r"^\s*uint64_t ([^;]*);", block, re.M):
        for name, count in re.findall(r"(\w+)(?:\[(\w+)\])?", line):
            depths[name] = {"": 1, "kVecSlots": SLOTS}.get(count) or int(count)
    return depths


class Model:
    def __init__(self, items, large):
        self.items, self.large = items, large   # items: (first of its q-tile, last of it, steps)
        self.depth = _depths()
        mma = ["mma"] if large else ["rows", "u", "ds"]
        self.count = {"tile_full": 1, "tile_free": len(mma) + 2, "vec_full": 1, "vec_empty": 2, "r_ready": 1, "s_free": 2,
                      "p_ready": 2, "ds_ready": 2, "qdo_ready": 2, "dq_free": 2}
        self.bars = {}      # (name, index) -> [arrivals of this phase, phases complete, clock of the arrivals so far, clock]
        self.log = {}       # buffer -> [(agent, time) of the last write, {agent: time} of the reads since]
        programs = {"softmax0": self.softmax(0), "softmax1": self.softmax(1), "fold0": self.fold(0), "fold1": self.fold(1),
                    "loader": self.loader()}
        programs.update({name: self.issuer(name) for name in mma})
        if large:
            programs["r"] = self.form_r()
        self.programs = programs
        self.queues = {name: [] for name in mma + ["loader"]}   # issued and not finished: operations with the issuer's clock
        self.clock = {a: {} for a in list(programs) + ["async " + q for q in self.queues]}
        self.pending = {a: None for a in programs}              # the operation a role stands at
        self.done = {a: 0 for a in programs}

    # ---- the kernel's roles.  at(name, n): the barrier of step n and the phase that step n completes
    def at(self, name, n):
        d = self.depth[name]
        return name, n % d, n // d

    def free(self, name, n):
        """... of the use before step n's of the same buffer"""
        name, i, phase = self.at(name, n)
        return name, i, phase - 1

    def walk(self):
        n = runs = batches = 0
        for it, (first, last, steps) in enumerate(self.items):
            yield it, n, runs, batches, first, last, steps
            n, runs, batches = n + steps, runs + last, batches + -(-steps // BATCH)

    def softmax(self, wg):
        for it, n0, runs, _, first, last, steps in self.walk():
            yield "wait", [("tile_full", 0, it)]
            yield "read", f"item{it % 4}"
            if first:
                yield "write", f"tmem {'Q dO'.split()[wg]}"
                yield "arrive", ("qdo_ready", 0)
            for n in range(n0, n0 + steps):
                yield "wait", [self.at("s_ready", n)]
                yield "read", f"S{wg}"
                yield "wait", [("acc_done", 1, n - 1)]
                yield "write", f"P{wg}"
                yield "wait", [self.at("dp_ready", n), self.free("ds_free", n)]
                yield "read", f"dP{wg}"
                yield "read", f"S{wg}"
                yield "arrive", self.at("s_free", n)
                yield "write", f"P{wg}"
                yield "write", f"dS{n % 2}{wg}"
                yield "arrive", self.at("p_ready", n)
                yield "read", f"dP{wg}"
                yield "write", f"dS{n % 2}{wg}"
                yield "arrive", self.at("ds_ready", n)
            if last:
                yield "wait", [("dq_done", 0, runs)]
                yield "read", f"dQ{wg}"
                yield "arrive", ("dq_free", 0)

    def fold(self, role):
        raw = ("K1 tile", "SiLU tile")[role]
        ready, free = (("a_ready", "a_free"), ("ap_ready", "ap_free"))[role]
        ahead = 1 if self.large and role else 2
        for it, n0, _, b0, _, _, steps in self.walk():
            yield "wait", [("tile_full", 0, it)]
            yield "read", f"item{it % 4}"
            yield "read", raw
            yield "arrive", ("tile_free", 0)
            for i0 in range(steps + ahead):
                if i0 < steps:
                    m, b = n0 + i0, b0 + i0 // BATCH
                    single = self.large and role
                    waits = [(free, (m - 1) % 2, (m - 1) // 2) if single else self.free(free, m)]
                    if i0 % BATCH == 0:
                        waits.append(self.at("vec_full", b))
                    yield "wait", waits
                    yield "read", f"rows{b % SLOTS}"
                    yield "write", self.operand(role, m)
                    yield "arrive", (ready, 0) if single else self.at(ready, m)
                i = i0 - ahead
                if i >= 0:
                    yield "wait", [("acc_done", role, n0 + i)]
                    yield "read", f"rows{(b0 + i // BATCH) % SLOTS}"
                    yield "read", "GU"[role]
                    yield "arrive", ("acc_free", role)
                    if i % BATCH == BATCH - 1 or i == steps - 1:
                        yield "arrive", self.at("vec_empty", b0 + i // BATCH)

    def operand(self, role, m):
        """The buffer of A (role 0) or A' (role 1) of step m."""
        if role == 0:
            return f"A{m % 2}"
        return "A'" if self.large or m % 2 == 0 else "SiLU tile"

    def form_r(self):
        for it, n0, _, b0, _, _, steps in self.walk():
            yield "wait", [("tile_full", 0, it)]
            yield "read", f"item{it % 4}"
            yield "read", "Q tile"
            yield "wait", [("ap_ready", 0, n0)]
            for i in range(steps):
                if i % BATCH == 0:
                    yield "wait", [self.at("vec_full", b0 + i // BATCH)]
                if i > 0:
                    yield "wait", [self.at("s_ready", n0 + i - 1)]
                yield "read", f"rows{(b0 + i // BATCH) % SLOTS}"
                yield "read", "Q tile"
                yield "write", "SiLU tile"
                yield "arrive", self.at("r_ready", n0 + i)

    def issuer(self, who):
        rows, u, ds = (who in ("mma", x) for x in ("rows", "u", "ds"))
        product = lambda reads, writes, *commits: ("issue", reads, writes, commits)

        def issue_s(m):
            yield "wait", [self.at("r_ready", m) if self.large else self.at("a_ready", m), self.free("s_free", m)]
            yield product(["SiLU tile", "K1 tile"] if self.large else [self.operand(0, m), "tmem Q"], ["S0", "S1"], self.at("s_ready", m))

        def issue_dp(m, after):
            yield "wait", [("ap_ready", 0, m) if self.large else self.at("ap_ready", m)] + ([self.at("ds_ready", m - 1)] if after else [])
            yield product([self.operand(1, m), "tmem dO"], ["dP0", "dP1"], self.at("dp_ready", m), ("ap_free", m % 2))

        for it, n0, runs, _, first, last, steps in self.walk():
            yield "wait", [("tile_full", 0, it)]
            yield "read", f"item{it % 4}"
            if first:
                yield "wait", [("qdo_ready", 0, runs)]
            if rows:
                yield from issue_s(n0)
                yield from issue_dp(n0, False)
            for n in range(n0, n0 + steps):
                more = n + 1 < n0 + steps
                if rows and more:
                    yield from issue_s(n + 1)
                    if not self.large:
                        yield from issue_dp(n + 1, True)
                if u:
                    yield "wait", [self.at("p_ready", n), ("acc_free", 1, n - 1)]
                    yield product(["P0", "P1", "dO tile"], ["U"], ("acc_done", 1))
                if ds:
                    yield "wait", [self.at("ds_ready", n)]
                    if self.large and more:
                        yield from issue_dp(n + 1, True)
                    if n == n0 and first:
                        yield "wait", [("dq_free", 0, runs - 1)]
                    if self.large:
                        yield "wait", [self.at("a_ready", n)]
                    grads = [f"dS{n % 2}0", f"dS{n % 2}1"]
                    yield product(grads + [self.operand(0, n)], ["dQ0", "dQ1"], self.at("a_free", n))
                    yield "wait", [("acc_free", 0, n - 1)]
                    yield product(grads + ["Q tile"], ["G"], ("acc_done", 0), self.at("ds_free", n))
            yield product([], [], ("tile_free", 0), *([("dq_done", 0)] if ds and last else []))

    def loader(self):
        for it, _, _, b0, first, _, steps in self.walk():
            yield "wait", [("tile_free", 0, it - 1)]
            yield "write", f"item{it % 4}"
            yield "issue", [], ["K1 tile", "SiLU tile"] + (["Q tile", "dO tile"] if first else []), [("tile_full", 0)]
            for b in range(b0, b0 + -(-steps // BATCH)):
                yield "wait", [self.free("vec_empty", b)]
                yield "issue", [], [f"rows{b % SLOTS}"], [self.at("vec_full", b)]

    # ---- running them
    def bar(self, name, index):
        return self.bars.setdefault((name, index), [0, 0, {}, {}])

    @staticmethod
    def join(a, b):
        for k, v in b.items():
            a[k] = max(a.get(k, 0), v)

    def touch(self, agent, buffer, write):
        clock = self.clock[agent]
        clock[agent] = clock.get(agent, 0) + 1
        last, reads = self.log.setdefault(buffer, [None, {}])
        for other, t in ([last] if last else []) + (list(reads.items()) if write else []):
            assert clock.get(other, 0) >= t, f"{agent} {'writes' if write else 'reads'} {buffer}, not ordered behind {other}"
        if write:
            self.log[buffer] = [(agent, clock[agent]), {}]
        else:
            reads[agent] = clock[agent]

    def arrive(self, agent, name, index, *_):
        b = self.bar(name, index)
        self.join(b[2], self.clock[agent])
        b[0] += 1
        if b[0] == self.count.get(name, 1):
            b[0], b[1] = 0, b[1] + 1
            self.join(b[3], b[2])

    def ready(self, role):
        if self.pending[role] is None:
            self.pending[role] = next(self.programs[role], ("end",))
        op = self.pending[role]
        if op[0] == "end":
            return False
        return op[0] != "wait" or all(self.bar(name, i)[1] % 2 != phase % 2 for name, i, phase in op[1])

    def step(self, role):
        op, self.pending[role] = self.pending[role], None
        self.done[role] += 1
        if op[0] == "wait":
            for name, i, phase in op[1]:
                assert self.bar(name, i)[1] > phase, f"{role} passes {name} before its phase {phase} is complete"
                self.join(self.clock[role], self.bar(name, i)[3])
        elif op[0] == "issue":
            self.queues[role].append((op[1:], dict(self.clock[role])))
        elif op[0] == "arrive":
            self.arrive(role, *op[1])
        else:
            self.touch(role, op[1], op[0] == "write")

    def finish(self, queue):
        (reads, writes, commits), clock = self.queues[queue].pop(0)
        agent = "async " + queue
        self.join(self.clock[agent], clock)
        for buffers, write in ((reads, False), (writes, True)):
            for b in buffers:
                self.touch(agent, b, write)
        for c in commits:
            self.arrive(agent, *c)

    def moves(self):
        return [(self.step, r) for r in self.programs if self.ready(r)] + [(self.finish, q) for q in self.queues if self.queues[q]]

    def run(self, held=None, at=0, rng=None):
        """held: this role stands still before its operation `at` until nothing else can move."""
        released = held is None
        turn = 0
        while True:
            moves = self.moves()
            if not released:
                others = [m for m in moves if m[1] != held or m[0] == self.finish or self.done[held] < at]
                released = not others
                moves = others or moves
            if not moves:
                break
            do, who = rng.choice(moves) if rng else moves[turn % len(moves)]
            do(who)
            turn += 1
        stuck = {r: (self.done[r], op) for r, op in self.pending.items() if op[0] != "end"}
        assert not stuck, f"{held} held back at {at}: waiting for ever: {stuck}"


ITEMS = [(1, 0, 3), (0, 1, 5), (1, 1, 1), (1, 0, 1), (0, 1, 2)]   # (first of its q-tile, last of it, steps)


@pytest.mark.parametrize("large", [False, True])
def test_no_order_of_the_roles_hangs_or_races(large):
    model = Model(ITEMS, large)
    model.run()
    for role, operations in model.done.items():
        for at in range(operations):
            Model(ITEMS, large).run(role, at)
    for seed in range(40):
        rng = random.Random(seed)
        Model([(1, 0, rng.randint(1, 9)), (0, 1, rng.randint(1, 9)), (1, 1, rng.randint(1, 6))], large).run(rng=rng)


def test_the_model_sees_a_barrier_two_phases_ahead():
    """ds_ready as a single barrier (a mistake planted in the model): the warp that issues dQ and G misses a phase."""
    def run(role, at):
        model = Model(ITEMS, False)
        model.depth["ds_ready"] = 1
        model.run(role, at)

    operations = Model(ITEMS, False)
    operations.run()
    with pytest.raises(AssertionError, match="waiting for ever.*ds_ready"):
        for at in range(operations.done["ds"]):
            run("ds", at)

"""Host-only models of the kernels' barrier protocols, run under adversarial schedules.

A kernel's roles (TMA producer, product issuer, compute and drain warps, ...) are written down as generators of
what they execute, in the order of the CUDA source:

    ("wait", barrier, k)        parity wait for the barrier's k-th completion, counted from 0
    ("arrive", barrier)
    ("tma", barrier, writes)    a load: after any delay and in any order its writes appear and it arrives
    ("mma", reads, writes)      a product, queued behind the issuer's earlier ones; reads and writes when it runs
    ("commit", barrier)         an arrival once the issuer's products so far have run, after any further delay
    ("read", cell, tag), ("write", cell, tag)
    ("bulk", reads)             a store or reduce-add out of shared memory: reads after any delay
    ("bulk_wait", n)            until all but the n youngest of those have read
    ("sync", name, n)           a named barrier of n roles
    ("any", name, n, flag)      the same with a reduction: yields whether any of the n flags was set
    ("settle", barrier, k)      a wait that does not look at the abort flag (for copies and products on their way)

A role that is several warps is several agents, each with its own part of the data and its own arrivals
(`need`: arrivals per phase): one agent for all of them would hide that they can be a tile apart.

Two things are checked. A parity wait is only right while its barrier has seen k or k + 1 completions: further
ahead it blocks for ever (on the GPU until the bounded wait expires), behind it passes too early. And every cell
(a tile in shared memory, columns of tensor memory) carries a tag for its contents: whoever reads names the tag
that must be there. A product or store reads when it runs, which may be long after it was issued.

When the last agent has come to its end the CTA retires: no load may be on its way and no product at work.

With `abort` one wait of the run gives up as if its bound had been reached. From there on every wait that is not
ready fails, as it does once the CTA's abort flag is up (the agent sees `Aborted`), contents are no longer
checked, and what has to hold is that every agent comes to its end.
"""


class Violation(Exception):
    pass


class Aborted(Exception):
    """Thrown into an agent whose wait gave up."""


class Model:
    need: dict = {}   # arrivals per phase, by the barrier's name up to its index; default 1

    def __init__(self, rng, abort=False):
        self.rng = rng
        self.done, self.count = {}, {}    # completed phases, arrivals in the current one
        self.cells = {}
        self.tma, self.bulk, self.loads = [], [], {}   # loads: how many each barrier has been given
        self.queues = {}
        self.syncs = {}                   # name -> [completed generations, arrivals, flags so far, last result]
        self.aborted = False
        self.abort_after = rng.randrange(1, 1200) if abort else None

    def agents(self):
        raise NotImplementedError

    # ---- how issuing threads leave ----
    def producing(self, body):
        """A producer's loads are waited for at its end, whether or not one of its waits gave up."""
        try:
            yield from body
        except Aborted:
            pass
        for bar, n in sorted(self.loads.items()):
            yield ("settle", bar, n - 1)

    def issuing(self, body, bar="settled"):
        """And an issuer's products, by a barrier that nothing else uses."""
        try:
            yield from body
        except Aborted:
            pass
        yield ("commit", bar)
        yield ("settle", bar, 0)

    # ---- primitives ----
    def arrive(self, name):
        self.count[name] = self.count.get(name, 0) + 1
        if self.count[name] == self.need.get(name.split("[")[0], 1):
            self.count[name] = 0
            self.done[name] = self.done.get(name, 0) + 1

    def check(self, reads):
        if self.aborted:
            return
        for cell, tag in reads:
            if self.cells.get(cell) != tag:
                raise Violation(f"{cell} holds {self.cells.get(cell)}, {tag} expected")

    def ready(self, op):
        if op[0] in ("wait", "settle"):
            c = self.done.get(op[1], 0)
            if c - op[2] not in (0, 1) and not self.aborted:
                raise Violation(f"{op[1]}: waiter wants completion {op[2]}, barrier has completed {c}")
            return (c - op[2]) % 2 == 1   # the parity that the hardware looks at
        if op[0] == "bulk_wait":
            return all(b is None for b in self.bulk[:max(0, len(self.bulk) - op[1])])
        return self.syncs[op[1]][0] > op[2]   # sync, any: op[2] is the generation it joined

    def issue(self, who, op):
        """Executes an operation; returns it if the agent has to wait for it."""
        kind = op[0]
        if kind in ("wait", "bulk_wait", "settle"):
            return op
        if kind in ("sync", "any"):
            state = self.syncs.setdefault(op[1], [0, 0, False, False])
            joined = state[0]
            state[1] += 1
            state[2] |= kind == "any" and op[3]
            if state[1] == op[2]:
                state[:] = joined + 1, 0, False, state[2]
            return (kind, op[1], joined)
        if kind == "arrive":
            self.arrive(op[1])
        elif kind == "tma":
            self.tma.append((op[1], op[2] if len(op) > 2 else []))
            self.loads[op[1]] = self.loads.get(op[1], 0) + 1
        elif kind in ("mma", "commit"):
            self.queues.setdefault(who, []).append(op)
        elif kind == "read":
            self.check([op[1:]])
        elif kind == "write":
            self.cells[op[1]] = op[2]
        elif kind == "bulk":
            self.bulk.append(op[1])
        else:
            raise ValueError(op)
        return None

    def run_async(self, where):
        if where == "tma":
            name, writes = self.tma.pop(self.rng.randrange(len(self.tma)))
            self.cells.update(writes)
            self.arrive(name)
        elif where == "bulk":
            at = self.rng.choice([i for i, b in enumerate(self.bulk) if b is not None])
            self.check(self.bulk[at])
            self.bulk[at] = None
        else:
            op = self.queues[where].pop(0)
            if op[0] == "commit":
                self.arrive(op[1])
            else:
                self.check(op[1])
                self.cells.update(op[2])

    # ---- scheduler: anything that can move may be next; one party at a time is slowed down heavily ----
    def run(self, max_steps=400000):
        agents = self.agents()
        pending = {n: None for n in agents}
        alive = set(agents)
        parties = list(agents) + ["tma", "bulk"]
        slow = self.rng.choice(parties)
        for step in range(max_steps):
            movable, failing = [], []
            for n in sorted(alive):   # a fixed order, so that a seed names one schedule
                op = pending[n]
                if op is None or self.ready(op):
                    movable.append(n)
                elif op[0] == "wait":
                    failing.append(n)
            if self.abort_after is not None and step >= self.abort_after and failing:
                self.aborted = True
            if self.aborted:
                movable += failing
            if self.tma:
                movable.append("tma")
            if any(b is not None for b in self.bulk):
                movable.append("bulk")
            movable += ["queue " + q for q, ops in sorted(self.queues.items()) if ops]
            if not movable:
                if alive:
                    raise Violation(f"stuck: { {n: pending[n][1:] for n in sorted(alive)} }")
                return
            who = self.rng.choice(movable)
            if who == slow and self.rng.random() < 0.9 and len(movable) > 1:
                continue
            if self.rng.random() < 0.02:
                slow = self.rng.choice(parties)
            if who not in agents:
                self.run_async(who.removeprefix("queue "))
                continue
            failed, before = who in failing, pending[who]
            pending[who] = None
            try:
                if failed:
                    op = agents[who].throw(Aborted())
                elif before is not None and before[0] == "any":
                    op = agents[who].send(self.syncs[before[1]][3])
                else:
                    op = next(agents[who])
            except (StopIteration, Aborted):
                alive.discard(who)
                if not alive and (self.tma or any(op[0] == "mma" for q in self.queues.values() for op in q)):
                    raise Violation("loads or products at work at the exit") from None
                continue
            pending[who] = self.issue(who, op)
        raise Violation("did not finish")


def survives(make, seeds):
    """Runs make(seed) for every seed; the first violation, with its seed, or None."""
    for seed in seeds:
        try:
            make(seed).run()
        except Violation as e:
            return seed, str(e)
    return None

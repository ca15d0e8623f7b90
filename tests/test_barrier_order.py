"""CPU: no wait of the warp-specialised kernels rests on timing.

An mbarrier is waited for by the parity of a phase: the wait has to be made before the NEXT phase of the barrier completes, or it blocks on the phase
after that.  So for every wait something must keep the next phase from completing until the waiter has passed.  The roles of the kernels that carry
the state, of the WY preparation and of the chunk backward are restated here as sequences of arrivals and waits; every role is held in front of each of its waits while all
others run as far as they can (copies and products complete at once), and the barrier it is held at must not have gone past the phase it waits for.
The system is monotone, so this covers every schedule.

How many barriers stand behind a name (one per buffer slot, or one in all) is read from the kernels' shared structs.  Warps that act alike are two
agents, so that one of them may be late.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mogankda_b200", "csrc")
STEPS = 7


def _slots(source, struct):
    """{barrier: barriers per chain or item} of the uint64_t members of a kernel's shared struct."""
    text = open(os.path.join(CSRC, source)).read()
    body = re.search(r"struct %s \{(.*?)\n\};" % struct, text, re.S)[1]
    found = {}
    for line in re.findall(r"uint64_t ([^;]*);", body):
        for name, dims in re.findall(r"(\w+)((?:\[\d+\])*)", line):
            found[name] = [int(d) for d in re.findall(r"\d+", dims)]
    return found


class Roles:
    """Agents: name -> [("wait" | "arrive", barrier, phase)].  `slots`: barriers behind a name that takes a step number."""

    def __init__(self, slots):
        self.slots, self.count, self.agents = slots, {}, {}

    def at(self, name, k):
        n = self.slots.get(name, 1)
        return (name, k % n), k // n

    def agent(self, name):
        ops = self.agents.setdefault(name, [])

        def wait(bar, k):
            ops.append(("wait", *self.at(bar, k)))

        def arrive(bar, k):
            ops.append(("arrive", self.at(bar, k)[0], None))
        return wait, arrive

    def run(self, held=None, at=None):
        """Arrivals per barrier when nobody can go on; every agent has to come to its end if none is held."""
        pos, got = dict.fromkeys(self.agents, 0), {}
        moved = True
        while moved:
            moved = False
            for name, ops in self.agents.items():
                while pos[name] < len(ops) and not (name == held and pos[name] == at):
                    what, bar, phase = ops[pos[name]]
                    if what == "wait":
                        if got.get(bar, 0) // self.count.get(bar[0], 1) <= phase:
                            break
                    else:
                        got[bar] = got.get(bar, 0) + 1
                    pos[name] += 1
                    moved = True
        if held is None:
            assert all(pos[n] == len(ops) for n, ops in self.agents.items()), {n: ops[pos[n]] for n, ops in self.agents.items() if pos[n] < len(ops)}
        return got

    def late_waits(self):
        """The waits that could be made too late: (agent, barrier)."""
        self.run()
        bad = set()
        for name, ops in self.agents.items():
            for i, (what, bar, phase) in enumerate(ops):
                if what == "wait" and not bar[0].startswith("sync"):
                    if self.run(name, i).get(bar, 0) // self.count.get(bar[0], 1) > phase + 1:
                        bad.add((name, bar[0]))
        return sorted(bad)


def pair(dims, n=STEPS):
    """recur_fwd_pair: two chains (0: state, 1: transition) with common tiles, all double-buffered."""
    slots = {}
    for name in ("fullN", "fullK", "fullU", "uFree"):
        slots[name] = dims[name][0] if dims[name] else 1
    for name in ("opS", "opV", "mm1", "mm2"):
        for c in range(2):
            slots[f"{name}{c}"] = dims[name][1] if len(dims[name]) > 1 else 1
    r = Roles(slots)
    r.count = {"uFree": 2, **{f"op{x}{c}": 2 for x in "SV" for c in range(2)}}
    wait, arrive = r.agent("load")

    def load(bar, k):
        if k < n:
            arrive(bar, k)
    for k in range(2):
        load("fullU", k), load("fullN", k), load("fullK", k)
    for k in range(n):
        wait("uFree", k), load("fullU", k + 2)
        wait("mm11", k), load("fullN", k + 2)
        wait("mm21", k), load("fullK", k + 2)
    wait, arrive = r.agent("mma")
    for k in range(n):
        wait("fullN", k)
        for c in "01":
            wait("opS" + c, k), arrive("mm1" + c, k)
        wait("fullK", k)
        for c in "01":
            wait("opV" + c, k), arrive("mm2" + c, k)
    for c in "01":
        for w in "ab":
            wait, arrive = r.agent(f"chain{c}{w}")

            def preload_u(k):
                if c == "0" and k < n:
                    wait("fullU", k), arrive("uFree", k)
            preload_u(0)
            for k in range(n):
                wait("fullN", k)
                if k:
                    wait("mm2" + c, k - 1)
                arrive("opS" + c, k)
                wait("mm1" + c, k)
                arrive("opV" + c, k)
                preload_u(k + 1)
            wait("mm2" + c, n - 1)
    return r


def chain(dims, out, norm=False, save_h=False, n=STEPS):
    """recur_fwd (out = False: every tile double-buffered) and chain_fwd (one buffer each; without a norm and without states to save two of nw^T)."""
    late = out and not norm
    D = 1 if out else 2
    dn = 2 if D == 2 or (late and not save_h) else 1
    slots = {k: (d[0] if d else 1) for k, d in dims.items()}
    slots.update(fullN=dn, fullK=D, fullU=D, ready=1, freed=1)
    r = Roles(slots)
    r.count = {"opS": 2, "opV": 2, "uFree": 2, "oFree": 2, "gFree": 2, "ready0": 2, "ready1": 2}
    wait, arrive = r.agent("load")

    def load(bar, k):
        if k < n:
            arrive(bar, k)
    load("fullU", 0), load("fullN", 0), load("fullK", 0)
    if out:
        load("fullQ", 0), load("fullA", 0)
    if dn > 1:
        load("fullN", 1)
    if D > 1:
        load("fullU", 1), load("fullK", 1)
    wait("uFree", 0), load("fullU", D)
    for k in range(n):
        wait("mm1", k), load("fullN", k + dn)
        if k + 1 < n and D > 1:
            wait("uFree", k + 1), load("fullU", k + 1 + D)
        wait("mm2", k), load("fullK", k + D)
        if out:
            if late and k + 1 < n:
                wait("uFree", k + 1), load("fullU", k + 2)
            wait("mmS", k), load("fullQ", k + 1)
            wait("mmO", k), load("fullA", k + 1)
            if not late and k + 1 < n:
                wait("uFree", k + 1), load("fullU", k + 2)
    wait, arrive = r.agent("mma")

    def output(k):
        wait("fullQ", k)
        if k:
            wait("oFree", k - 1)
        arrive("mmS", k)
    for k in range(n):
        wait("fullN", k), wait("opS", k), arrive("mm1", k)
        if out and not late:
            output(k)
        wait("fullK", k), wait("opV", k), arrive("mm2", k)
        if out:
            if late:
                output(k)
            wait("fullA", k), arrive("mmO", k)
    if out:
        for w in "ab":
            wait, arrive = r.agent("epilogue" + w)
            for k in range(n):
                if norm:
                    wait("fullG", k)
                wait("mmO", k), arrive("oFree", k), arrive("gFree", k)
        if norm:
            wait, arrive = r.agent("gate")
            for k in range(n):
                if k:
                    wait("gFree", k - 1)
                arrive("fullG", k)
        if save_h:
            wait, arrive = r.agent("store")
            for k in range(n):
                for hf in "01":
                    wait("ready" + hf, k), arrive("freed" + hf, k)
    for w in "ab":
        wait, arrive = r.agent("state" + w)

        def preload_u(k):
            wait("fullN", k), wait("fullU", k), arrive("uFree", k)
        preload_u(0)
        for k in range(n):
            if k:
                wait("mm2", k - 1)
                if late:
                    wait("mmS", k - 1)
            arrive("opS", k)
            if save_h:
                if k:
                    wait("freed1", k - 1)
                arrive("ready0", k)
            wait("mm1", k)
            arrive("opV", k)
            if save_h:
                wait("freed0", k), arrive("ready1", k)
            if k + 1 < n:
                preload_u(k + 1)
        wait("mm2", n - 1)
    return r


def reverse(dims, n=STEPS):
    """bwd_dh."""
    r = Roles({k: (d[0] if d else 1) for k, d in dims.items()})
    r.count = {"opS": 2, "opV": 2}
    wait, arrive = r.agent("load")
    arrive("fullA", 0), arrive("fullK", 0), arrive("fullN", 0), arrive("fullA", 1)
    for k in range(n - 1):
        wait("mm1", k), arrive("fullK", k + 1)
        wait("mm2", k), arrive("fullN", k + 1)
        if k + 2 < n:
            arrive("fullA", k + 2)
    wait, arrive = r.agent("mma")
    wait("fullA", 0)
    for k in range(n):
        wait("fullK", k), wait("opS", k), arrive("mm1", k)
        wait("fullN", k), wait("opV", k), arrive("mm2", k)
        if k + 1 < n:
            wait("fullA", k + 1)
    for w in "ab":
        wait, arrive = r.agent("state" + w)
        for k in range(n):
            if k:
                wait("mm2", k - 1)
            arrive("opS", k)
            wait("fullA", k), wait("mm1", k), arrive("opV", k)
        wait("mm2", n - 1)
    return r


def intra(dims, dtype, scalar, n=STEPS):
    """intra_fwd: X and Y on neighbouring items, two threads that issue products, two that copy."""
    late_q = dtype == "fp32" and not scalar
    slots = {k: (d[0] if d else 1) for k, d in dims.items()}
    slots["op1"] = 1                                       # [2] are the halves of the channels
    r = Roles(slots)
    x_bars, y_bars = ("op1h0", "op1h1", "rows", "hand", "nwReady", "uReady", "syncA", "syncB"), ("opA", "opV", "acc", "syncY", "syncI")
    r.count = {**dict.fromkeys(x_bars, 2), **dict.fromkeys(y_bars, 2), "ldin": 2}
    for w in "ab":
        wait, arrive = r.agent("X" + w)

        def read_out(k):
            wait("mmN", k), arrive("nwReady", k)
            wait("mmU", k), arrive("uReady", k)
        for k in range(n):
            wait("ldin", k)
            if not scalar and k:
                wait("hand", k - 1)
            arrive("syncA", k), wait("syncA", k)
            if not scalar and k:
                wait("khFree", k - 1)
            arrive("op1h0", k), arrive("op1h1", k)
            if scalar and k:
                wait("khFree", k - 1)
            arrive("syncB", k), wait("syncB", k)
            arrive("rows", k)
            if k:
                read_out(k - 1)
            wait("mm1", k), wait("rows", k)
            if k:
                wait("bkFree", k - 1)
            arrive("hand", k)
        read_out(n - 1)
        wait, arrive = r.agent("Y" + w)
        for k in range(n):
            wait("rows", k), wait("mm1", k)
            arrive("acc", k)
            arrive("syncY", k), wait("syncY", k)
            if k:
                wait("abFree", k - 1)
            arrive("syncI", k), wait("syncI", k)
            if dtype != "fp32":
                wait("fullV", k)
            arrive("opA", k)
            wait("mmV", k), arrive("opV", k)
    wait, arrive = r.agent("products X")
    for k in range(n):
        wait("op1h0", k), wait("op1h1", k), arrive("mm1", k)
    wait, arrive = r.agent("products Y")
    for k in range(n):
        wait("hand", k), wait("opA", k)
        arrive("mmV", k)
        if k + 1 == n:
            arrive("mmN", k)
        wait("opV", k), arrive("mmU", k)
        if k + 1 < n:
            arrive("mmN", k)
    wait, arrive = r.agent("copies X")

    def load_rows(k):
        if k < n:
            arrive("ldin", k)
            if not late_q:
                arrive("ldin", k)
    load_rows(0)
    if late_q:
        arrive("ldin", 0)
    for k in range(n):
        wait("mm1", k), load_rows(k + 1)
        wait("acc", k), wait("hand", k)
        arrive("khFree", k)
        if late_q and k + 1 < n:
            arrive("ldin", k + 1)
    wait, arrive = r.agent("copies Y")
    if dtype != "fp32":
        arrive("fullV", 0)
    for k in range(n):
        wait("nwReady", k), wait("uReady", k)
        arrive("bkFree", k), arrive("abFree", k)
        if dtype != "fp32" and k + 1 < n:
            arrive("fullV", k + 1)
    return r


def test_a_wait_that_rests_on_timing_is_found():
    """The pair kernel with one barrier in all for u^T used and for each product: the copying thread may come to its waits two phases late."""
    dims = dict(fullN=[2], fullK=[2], fullU=[2], uFree=[], opS=[2], opV=[2], mm1=[2], mm2=[2])
    assert ("load", "uFree") in pair(dims).late_waits()


def test_recur_fwd_pair():
    assert pair(_slots("tc_recur.cu", "Shared")).late_waits() == []


@pytest.mark.parametrize("out,norm,save_h", [(False, False, False), (True, True, False), (True, True, True), (True, False, False), (True, False, True)])
def test_recur_fwd_and_chain_fwd(out, norm, save_h):
    assert chain(_slots("tc_recur.cu", "RecurShared"), out, norm, save_h).late_waits() == []


def test_bwd_dh():
    assert reverse(_slots("tc_recur.cu", "DhShared")).late_waits() == []


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", ["fp16", "fp32"])
def test_intra_fwd(dtype, scalar):
    assert intra(_slots("tc_intra.cu", "Shared"), dtype, scalar).late_waits() == []


def bwd_chunk(dims, scalar, from_hbm, n=STEPS):
    """bwd_chunk: compute warps a (row block 0), b (row block 3), one thread that issues products, one that copies, one warp for the per-row scalars."""
    slots = {k: (d[0] if d else 1) for k, d in dims.items()}
    slots["mmI"] = slots["opI"] = 1                        # [4] are the row blocks
    r = Roles(slots)
    r.count = {**dict.fromkeys(("opW", "free", "opI3", "syncTop", "syncMid", "syncEnd"), 2), "fullS": 2}
    if scalar:
        r.count["opI0"] = 2
    for w in "ab":
        wait, arrive = r.agent("compute" + w)

        def sync(name, k):
            arrive(name, k), wait(name, k)
        for k in range(n):
            wait("rows", k)
            sync("syncTop", k)
            wait("mmW", k), arrive("opW", k)
            wait("fullS", k), wait("fullT", k), wait("mmL", k), wait("mmT", k)
            sync("syncMid", k)
            arrive("free", k)
            if scalar or w == "a":
                arrive("opI3", k) if not scalar else None
                arrive("opI0", k)
            else:
                arrive("opI3", k)
            wait("mmI0" if scalar or w == "a" else "mmI3", k)
            sync("syncEnd", k)
    wait, arrive = r.agent("products")
    wait("fullW", 0), arrive("mmW", 0)
    for k in range(n):
        wait("fullS", k), wait("opW", k), arrive("mmL", k)
        wait("fullT", k), arrive("mmT", k)
        if not scalar:
            wait("opI3", k), arrive("mmI3", k)
        wait("opI0", k), arrive("mmI0", k)
        if k + 1 < n:
            wait("mmI0", k), wait("fullW", k + 1), arrive("mmW", k + 1)
    wait, arrive = r.agent("copies")
    arrive("fullW", 0), arrive("fullS", 0)
    for k in range(n):
        if k:
            wait("mmI0", k - 1)
            if not scalar:
                arrive("fullW", k)
        arrive("fullS", k)                                 # dO: the second part of its bytes
        wait("mmW", k), arrive("fullT", k)
        if k + 1 == n:
            break
        if from_hbm:
            wait("mmL", k)
        wait("free", k)
        if scalar:
            arrive("fullW", k + 1)
        arrive("fullS", k + 1)
    wait, arrive = r.agent("rows")
    for k in range(n):
        if k:
            wait("free", k - 1)
        arrive("rows", k)
    return r


@pytest.mark.parametrize("from_hbm", [False, True])
@pytest.mark.parametrize("scalar", [False, True])
def test_bwd_chunk(scalar, from_hbm):
    """... and no role waits for a phase of a barrier without having waited for the one in front of it: a wait by parity would return at once if that
    were still to come."""
    r = bwd_chunk(_slots("tc_bwd_chunk.cu", "Shared"), scalar, from_hbm)
    assert r.late_waits() == []
    for name, ops in r.agents.items():
        seen = {}
        for what, bar, phase in ops:
            if what == "wait":
                assert phase == seen.get(bar, 0), (name, bar, phase)
                seen[bar] = phase + 1


def step(dims, n=STEPS):
    """step_fwd_vk: compute warps a and b, one warp that fetches what the items are and their states."""
    r = Roles({k: (d[0] if d else 1) for k, d in dims.items()})
    r.count = {"empty": 2}
    wait, arrive = r.agent("load")
    for k in range(n + 1):                                 # the last one says that there are no more
        if k >= 2:
            wait("empty", k - 2)
        arrive("known", k)
        if k < n:
            arrive("full", k)
    for w in "ab":
        wait, arrive = r.agent("compute" + w)
        wait("known", 0)
        for k in range(n):
            wait("full", k), arrive("empty", k), wait("known", k + 1)
    return r


def test_step_fwd_vk():
    dims = _slots("step.cu", "Shared")
    assert step(dims).late_waits() == []
    assert step({k: [] for k in dims}).late_waits() != []


def _step_with_a_failure(n, fails):
    """step_fwd_vk over n items with two compute warps.  `fails`: (agent, i): its i-th wait gives up; what can go on no more gives up too, except at the block-wide
    barrier, where it would hang.  Barriers go by parity, as they do.  Returns the waits made by each agent."""
    done, info, state, waits = {}, [None] * 4, {"gave_up": False}, {}

    def arrive(bar, count=1):
        done[bar] = done.get(bar, 0) + 1 / count

    def load():
        j = 0
        for it in range(n + 1):
            if j >= 2 and not (yield ("empty", j - 2)):
                break
            info[j & 3] = (j, it if it < n else -1)
            arrive(("known", j & 1))
            if it == n:
                break
            arrive(("full", j & 1))
            j += 1
        for i in (j - 2, j - 1):
            if i >= 0:
                yield ("full", i)

    def compute():
        def request(j):
            if not (yield ("known", j)):
                state["gave_up"] = True
                return -1
            assert info[j & 3][0] == j
            return info[j & 3][1]
        item = yield from request(0)
        yield "sync"
        j = 0
        while item >= 0 and not state["gave_up"]:
            assert item == j
            yield "sync"
            here = yield ("full", j)
            if here:
                arrive(("empty", j & 1), 2)
            else:
                state["gave_up"] = True
            item = yield from request(j + 1)
            yield "sync"
            j += 1

    agents = {"load": load(), "a": compute(), "b": compute()}
    at = {name: next(a) for name, a in agents.items()}

    def step(name, value):
        try:
            at[name] = agents[name].send(value)
        except StopIteration:
            del at[name]
    while at:
        moved = False
        for name in list(at):
            if at[name] == "sync":
                continue
            bar, k = at[name]
            if (name, waits.get(name, 0)) == fails:
                ok = False
            elif int(done.get((bar, k & 1), 0) + 1e-9) & 1 != (k >> 1) & 1:
                ok = True
            else:
                continue
            waits[name] = waits.get(name, 0) + 1
            step(name, ok)
            moved = True
        if not moved and all(at.get(w) == "sync" for w in "ab"):
            for w in "ab":
                step(w, None)
            moved = True
        if not moved:
            late = [name for name in at if at[name] != "sync"]
            assert late, f"{fails}: the compute warps disagree on the number of block-wide barriers: {at}"
            for name in late:
                waits[name] = waits.get(name, 0) + 1
                step(name, False)
    return waits


@pytest.mark.parametrize("n", [1, 2, 3, 7])
def test_step_fwd_vk_comes_to_its_end_when_a_wait_gives_up(n):
    """Whichever it is: no warp reads what an item is without having been told, all compute warps leave behind the same block-wide barrier, and what the kernel does
    hangs on no wait whose outcome it drops."""
    for name, waits in _step_with_a_failure(n, None).items():
        for i in range(waits):
            _step_with_a_failure(n, (name, i))
    code = open(os.path.join(CSRC, "step.cu")).read()
    assert "mbar_wait" in code and not re.findall(r"(?:[;{}]|(?<!\(void)\))\s*umma::mbar_wait\(", code)         # (void): it is over either way

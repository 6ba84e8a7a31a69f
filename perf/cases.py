"""Timed workloads of the framework, each through its public Python entry points.

A case is a dict of plain values; `prepare` makes what a program holds before the call,
`run` makes one pass, `work` gives the bytes and operations the pass cannot do without.
The kinds:

  mcs        one lattice advanced n MCS (SchedulerSCA, SchedulerSCABit, SchedulerDT, DB4)
  disorder   the same with quenched two-class disorder
  measure    the measurement loop: MCS chunks, roughness and correlator rows on the device
  correlate  one correlator measurement of a lattice against a tagged snapshot
  gram       the exact height Gram over stored snapshots
  batch      many replicas of uneven size advanced together, measured and taken home

Lattices come back as the handle's own device words (no copy) where a program would leave
them on the GPU, and as host words where they are small enough to be looked at each time.
"""
import numpy as np
import torch

import cudakpz_b200 as kpz

POP_SITES = 1 << 20  # lattices up to this many sites are popped to the host in a pass


def listed():
    return [
        # the benchmark's two rate pairs at its size; 50 MCS lie between two measurements of a
        # run near t = 500 on the default schedule, and are no multiple of a pass depth
        dict(name="scabit-16384-p1q0", kind="mcs", scheduler="scaBit", lx=14, ly=14, p=1.0, q=0.0, n=50),
        dict(name="scabit-16384-half", kind="mcs", scheduler="scaBit", lx=14, ly=14, p=0.5, q=0.5, n=50),
        # rates of many random planes: the pair the DT runs and the growth studies use
        dict(name="scabit-8192-p95q05", kind="mcs", scheduler="scaBit", lx=13, ly=13, p=0.95, q=0.05, n=20),
        # quenched binary disorder on a wide lattice, SchedulerSCA's default rate in class 0
        dict(name="sca-disorder-4096x2048", kind="disorder", scheduler="sca", lx=12, ly=11, p=0.95, q=0.0,
             p1=0.5, q1=0.1, fill=0.25, n=10),
        # the smallest lattice in use, SchedulerSCABit's default rates, a few steps at a time
        dict(name="scabit-256-default", kind="mcs", scheduler="scaBit", lx=8, ly=8, p=0.5, q=0.0, n=10),
        # random-sequential runs: the default inner scheme at a large and at a small size, the
        # faster scheme at a middle one
        dict(name="dt-dbsh-16384", kind="mcs", scheduler="dt", inner="dbsh", lx=14, ly=14, p=0.95, q=0.05, n=2),
        dict(name="dt-dbsh-1024", kind="mcs", scheduler="dt", inner="dbsh", lx=10, ly=10, p=0.95, q=0.05, n=5),
        dict(name="dt-dt-2048", kind="mcs", scheduler="dt", inner="dt", lx=11, ly=11, p=0.95, q=0.05, n=10),
        # the frontend's loop: advance, measure, with a correlator tag for the first half
        dict(name="measure-8192", kind="measure", scheduler="scaBit", lx=13, ly=13, p=0.5, q=0.5, n=100, every=10),
        # one measurement of the benchmark's lattice against a snapshot
        dict(name="correlate-16384", kind="correlate", lx=14, ly=14, steps=40),
        # the full Gram of 64 snapshots at the benchmark's size
        dict(name="gram-16384x64", kind="gram", lx=14, ly=14, snaps=64),
        # replicas of the batched configuration (256, 1024, 2048, 4096 squared in the ratio
        # 4:2:1:1, three rate pairs) run to t = n, W^2 of each, lattices taken home
        dict(name="batch-128", kind="batch", unit=16, lxmax=12, n=1000),
    ]


_RATES = [(1.0, 0.0), (0.5, 0.5), (0.5, 0.0), (0.95, 0.05), (0.95, 0.0), (0.9, 0.1), (0.75, 0.25), (1.0, 1.0)]


def draw(rng):
    def steps(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["mcs", "mcs", "mcs", "dt", "dt", "disorder", "measure", "correlate", "gram", "batch"])
    p, q = rng.choice(_RATES) if rng.random() < 0.75 else (round(rng.uniform(0.1, 1.0), 3), round(rng.uniform(0.0, 0.5), 3))
    if kind == "mcs":
        return dict(kind="mcs", scheduler=rng.choice(["scaBit", "scaBit", "sca"]), lx=rng.randint(8, 14),
                    ly=rng.randint(8, 13), p=p, q=q, n=steps(1, 64))
    if kind == "dt":
        if rng.random() < 0.2:
            return dict(kind="mcs", scheduler="db4", lx=rng.randint(8, 13), ly=rng.randint(8, 13), p=p, q=q, n=steps(1, 10))
        return dict(kind="mcs", scheduler="dt", inner=rng.choice(["dbsh", "dbsh", "dt", "db", "dtdbsh", "dbshrep"]),
                    lx=rng.randint(9, 13), ly=rng.randint(8, 13), p=p, q=q, n=steps(1, 10))
    if kind == "disorder":
        return dict(kind="disorder", scheduler=rng.choice(["sca", "scaBit", "dt"]), lx=rng.randint(9, 13),
                    ly=rng.randint(8, 12), p=p, q=q, p1=round(rng.uniform(0.1, 1.0), 3),
                    q1=round(rng.uniform(0.0, 0.5), 3), fill=round(rng.uniform(0.05, 0.95), 2), n=steps(1, 20))
    if kind == "measure":
        every = rng.randint(1, 20)
        return dict(kind="measure", scheduler=rng.choice(["scaBit", "sca", "dt"]), lx=rng.randint(9, 12),
                    ly=rng.randint(8, 12), p=p, q=q, n=every * rng.randint(2, 8) + rng.randint(0, every), every=every)
    if kind == "correlate":
        return dict(kind="correlate", lx=rng.randint(8, 14), ly=rng.randint(8, 13), steps=rng.randint(5, 40))
    if kind == "gram":
        return dict(kind="gram", lx=rng.randint(8, 13), ly=rng.randint(8, 13), snaps=rng.randint(2, 64))
    return dict(kind="batch", unit=rng.randint(1, 12), lxmax=rng.randint(10, 12), n=steps(10, 400))


class _Words:
    """A scheduler's device words for torch.as_tensor, which keeps this object and with it the
    scheduler (whose memory the words are) for as long as the tensor lives."""

    def __init__(self, s):
        self.owner = s
        self.__cuda_array_interface__ = {"shape": (s.size_words(),), "typestr": "<i4", "data": (s.devicePtr(), False),
                                         "version": 3}


def _lattice(s):
    if s.size() <= POP_SITES:
        return s.popSystem()
    return torch.as_tensor(_Words(s), device="cuda")


def _scheduler(case, seed):
    s = kpz.Scheduler(case["lx"], case["ly"], scheduler=case["scheduler"])
    s.supplySeed(seed)
    if "inner" in case:
        s.setDtInner(case["inner"])
    return s


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _surfaces(case, seed):
    """Heights (rows, L) of a periodic single-step surface grown from the flat one, half way
    and at the end of `steps` checkerboard steps of deposition at p = 1/2."""
    rows, L = 1 << case["ly"], 1 << case["lx"]
    g = _generator(seed)
    y = torch.arange(rows, device="cuda", dtype=torch.int32)[:, None]
    x = torch.arange(L, device="cuda", dtype=torch.int32)[None, :]
    odd = ((x + y) & 1).to(torch.int8)
    h = odd.clone()
    half = None
    for t in range(2 * case["steps"]):
        up = h + 1
        low = (torch.roll(h, 1, 0) == up) & (torch.roll(h, -1, 0) == up) & (torch.roll(h, 1, 1) == up) & (
            torch.roll(h, -1, 1) == up)
        low &= torch.randint(0, 2, h.shape, generator=g, device="cuda", dtype=torch.int8).bool()
        low &= odd == (t & 1)
        h = h + 2 * low.to(torch.int8)
        if t == case["steps"]:
            half = h
    return half, h


def _cbbit(h):
    """ENC_CBBIT words (kpz/systemSize.h:143-165) of the slopes of the heights h."""
    rows, L = h.shape
    weights = (1 << torch.arange(8, device=h.device)).to(torch.uint8)
    odd_row = (torch.arange(rows, device=h.device) & 1).bool()[:, None]
    quads = []
    for sub in (0, 1):
        for axis in (1, 0):
            s = ((h - torch.roll(h, 1, axis)) > 0).to(torch.uint8)
            bits = torch.where(odd_row, s[:, 1 - sub::2], s[:, sub::2])
            quads.append((bits.reshape(-1, 8) * weights).sum(1, dtype=torch.uint8))
    return torch.cat(quads).cpu().numpy().view(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("mcs", "disorder", "measure"):
        s = _scheduler(case, seed)
        # a surface in its growth regime; rates that use no random number would grow the same
        # one from every seed
        s.setPQ(*((case["p"], case["q"]) if 0.0 < case["p"] < 1.0 else (0.5, 0.5)))
        s.mcsPQSyncRng(20)
        s.setPQ(case["p"], case["q"])
        if kind == "disorder":
            g = _generator(seed)
            bits = torch.rand((s.size_words(), 16), generator=g, device="cuda") < case["fill"]
            place = torch.tensor([((i & 3) << 1) | ((i >> 2) << 3) for i in range(16)], device="cuda")
            words = (bits.long() << place).sum(1)
            s.setPQ(case["p1"], case["q1"], 1)
            s.setDisorder(words.cpu().numpy().astype(np.uint32))
        return {"case": case, "s": s}
    if kind == "correlate":
        s = kpz.Scheduler(case["lx"], case["ly"], scheduler="scaBit")
        half, end = _surfaces(case, seed)
        s.pushSystem(_cbbit(half))
        s.correlateTag()
        s.pushSystem(_cbbit(end))
        return {"case": case, "s": s}
    if kind == "gram":
        s = kpz.Scheduler(case["lx"], case["ly"], scheduler="scaBit")
        g = kpz.Gram(case["lx"], case["ly"], case["snaps"])
        s.supplySeed(seed)
        s.setPQ(0.5, 0.5)
        s.mcsPQSyncRng(8)
        s.setPQ(1.0, 0.0)
        for _ in range(case["snaps"]):
            s.mcsPQSyncRng(1)
            g.add_device(s.devicePtr())
        s.close()
        return {"case": case, "g": g}
    sizes = [lx for lx, count in ((8, 4), (10, 2), (11, 1), (12, 1)) if lx <= case["lxmax"]
             for _ in range(count * case["unit"])]
    rates = [((1.0, 0.0), (0.9, 0.1), (0.75, 0.25))[(i * 7 + i // 3) % 3] for i in range(len(sizes))]
    b = kpz.Batch(sizes, [r[0] for r in rates], [r[1] for r in rates], [seed * 4096 + i for i in range(len(sizes))])
    return {"case": case, "b": b}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mcs":
        state["s"].mcsPQSyncRng(case["n"])
        return _lattice(state["s"])
    if kind == "disorder":
        state["s"].mcsDisorder2SyncRng(case["n"])
        return _lattice(state["s"])
    if kind == "measure":
        s = state["s"]
        start = s.deviceMcs()
        rows = s.measureRun(start + case["n"], kpz.make_sampling("linear", interval=case["every"]), corr_start=start,
                            corr_stop=start + case["n"] // 2)
        return rows, _lattice(s)
    if kind == "correlate":
        r, ch, cs = state["s"].correlate()
        return np.array([r.w2] + r.h + [ch, cs])
    if kind == "gram":
        return state["g"].compute()
    b = state["b"]
    b.mcs(case["n"])
    w2 = b.roughness()
    return w2, np.concatenate([b.pop(i) for i in range(b.n)])


def exact(case, seed):
    """The correlator measurement from the heights themselves in 64 bits; the other kinds give
    whole numbers, or depend on a random stream that only the framework has."""
    if case["kind"] != "correlate":
        return None
    half, end = _surfaces(case, seed)
    slope = [[(h - torch.roll(h, 1, a)) > 0 for a in (0, 1)] for h in (half, end)]
    agree = sum(2 * (a == b).sum(dtype=torch.int64).item() - a.numel() for a, b in zip(*slope))
    # the walk's heights are relative to (0, -1)
    half = (half.to(torch.int16) - half[-1, 0]).double()
    end = (end.to(torch.int16) - end[-1, 0]).double()
    mean = end.mean().item()
    cross = (half * end).mean().item() - half.mean().item() * mean
    moments, power = [], end.clone()
    for _ in range(7):
        moments.append(power.mean().item())
        power *= end
    return np.array([moments[1] - mean * mean] + moments + [cross, agree / end.numel() / 2.0])


def work(case):
    """bytes: every lattice or snapshot read once and written once; flops: thread-level
    integer operations of the rule itself (32-bit logic on words of 32 sites for the
    checkerboard updates, per attempt for the random-sequential ones), 8-bit multiply-adds
    of one triangle for the Gram."""
    kind = case["kind"]
    if kind == "batch":
        sites = case["unit"] * sum(count << (2 * lx) for lx, count in ((8, 4), (10, 2), (11, 1), (12, 1))
                                   if lx <= case["lxmax"])
        return {"bytes": sites / 2 + sites / 4, "flops": sites / 32 * case["n"] * 40}
    sites = 1 << (case["lx"] + case["ly"])
    if kind == "correlate":
        return {"bytes": 2 * sites / 4, "flops": 2 * sites}
    if kind == "gram":
        return {"bytes": case["snaps"] * sites / 8, "flops": case["snaps"] * (case["snaps"] + 1) * sites}
    lattices = 2 if kind != "disorder" else 3
    if case["scheduler"] in ("dt", "db4"):
        ops = 18 * sites * case["n"]
    else:
        planes = max((0 if r in (0.0, 1.0) else 1 if r == 0.5 else 6)
                     for r in (case["p"], case["q"], case.get("p1", 0.0), case.get("q1", 0.0)))
        # masks and flips 7 (both kinds of flip 9), 7 more for each random plane
        ops = (7 + (2 if case["q"] else 0) + 7 * planes) * sites / 32 * case["n"]
    rows = case["n"] // case["every"] if kind == "measure" else 0
    return {"bytes": lattices * sites / 4 + rows * sites / 8, "flops": ops + 2 * sites * rows}

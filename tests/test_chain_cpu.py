"""The tile lists of the one-launch Newton-Schulz (``ops/chain.py``), interpreted on
the CPU: dependencies, coverage and the numbers they produce."""
import numpy as np
import pytest
import torch

from dmuon_b200.ops import chain as CH
from dmuon_b200.optim import newton_schulz as NS

COEFS = tuple(map(tuple, NS.DEFAULT_COEFFICIENTS))


def _spec(L, m0, n0, formulation="gram", restarts=(2,), coefs=COEFS, h=1.0, vec=False):
    dt = torch.float16 if formulation == "gram" else torch.bfloat16
    return CH.GroupSpec(L, m0, n0, dt, formulation, coefs, restarts if formulation == "gram" else (), h, vec)


def _interpret(specs, bn, inputs):
    """Run the list in order with fp64 arithmetic; every buffer starts as NaN, so a tile
    that is read before it was written, or never written, shows in the result."""
    ops, ent = CH.build_entries(specs, bn)
    buf = []
    for s, x in zip(specs, inputs):
        names = ("R", "P") if s.formulation == "direct" else ("R", "R2", "RP", "P", "Qa", "Qb")
        d = {n: np.full((s.L, s.m, s.m), np.nan) for n in names}
        d["X"], d["X2"] = x.copy(), np.full_like(x, np.nan)
        d["final"] = np.full_like(x, np.nan)
        d["parts"] = None
        buf.append(d)
    first = np.cumsum([0] + [s.L for s in specs])
    done = np.zeros(first[-1], dtype=np.int64)
    # what has to be finished before a product may start, per matrix: everything up to `after`
    finished_by_op = [{} for _ in range(first[-1])]

    def tile(s, d, pr, ns, per, is_sum, b, split, mirror, rows, cols, r0, r1, c0, c1):
        assert r0 < rows and c0 < cols
        if is_sum:
            v = d["parts"][b].sum(0)[r0:r1, c0:c1]
        else:
            A = d[pr.A][b].T if pr.a_mn else d[pr.A][b]
            B = d[pr.B][b].T if pr.b_mn else d[pr.B][b]
            lo, hi = (split * per * 64, min(A.shape[1], (split + 1) * per * 64)) if per else (0, A.shape[1])
            assert lo < hi
            v = A[r0:r1, lo:hi] @ B[c0:c1, lo:hi].T
        if ns > 1 and not is_sum:
            if d["parts"] is None or d["parts"].shape[1] != ns:
                d["parts"] = np.full((s.L, ns, rows, cols), np.nan)
            d["parts"][b, split, r0:r1, c0:c1] = v
        else:
            v = pr.alpha * v
            if pr.C is not None:
                v = v + pr.beta * d[pr.C][b][r0:r1, c0:c1]
            v = v + pr.diag * np.eye(rows, cols)[r0:r1, c0:c1]
            d[pr.out][b, r0:r1, c0:c1] = v
            if mirror:
                d[pr.out][b, c0:c1, r0:r1] = v.T

    for x, y, z, w in ent.astype(np.int64):
        op, mirror, split = x & 0xFF, (x >> 8) & 1, (x >> 16) & 0x7FFF
        mt, nt, b, ctr = y & 0xFFFF, (y >> 16) & 0xFFFF, z & 0xFFFF, (z >> 16) & 0xFFFF
        g, pr, ns, per, is_sum = ops[op]
        s, d = specs[g], buf[g]
        assert ctr == first[g] + b and done[ctr] >= w
        assert x >= 0
        rows = s.m if pr.symmetric else s.m0
        cols = s.m if pr.symmetric else s.n0
        tn, tm = CH._SUM_COLS if is_sum else bn, CH.tile_rows(bn)
        halves = [(nt, mirror)]
        if bn == CH.PAIR and (x >> 9) & 1:
            halves.append((nt + 1, (x >> 10) & 1))
        for nt, mirror in halves:
            r0, r1, c0, c1 = mt * tm, min(rows, mt * tm + tm), nt * tn, min(cols, nt * tn + tn)
            tile(s, d, pr, ns, per, is_sum, b, split, mirror, rows, cols, r0, r1, c0, c1)
            done[ctr] += CH.WARPS_PER_TILE * (2 if bn == CH.PAIR else 1)
        finished_by_op[ctr][op] = done[ctr]
    # a count in the list stands for whole products: w equals the count after `after` finished
    ends = {}
    for i, (g, pr, ns, per, is_sum) in enumerate(ops):
        ends[g] = ends.get(g, []) + [(i, ns > 1 and not is_sum)]
    for x, y, z, w in ent.astype(np.int64):
        op, ctr = x & 0xFF, (z >> 16) & 0xFFFF
        assert w == 0 or w in set(finished_by_op[ctr].values())
        assert w == 0 or max(o for o, c in finished_by_op[ctr].items() if c <= w) < op
    return [d["final"] for d in buf]


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("shapes,formulation", [
    ([(1, 64, 96)], "gram"), ([(2, 128, 128)], "gram"), ([(1, 136, 1040)], "gram"), ([(1, 2056, 72)], "gram"),
    ([(3, 264, 200)], "direct"), ([(1, 72, 1544)], "direct"),
    ([(2, 256, 128), (1, 128, 328), (2, 72, 64)], "gram"), ([(2, 1096, 600)], "gram"), ([(30, 264, 64)], "gram"),
])
def test_tile_list_computes_the_iteration(shapes, formulation, bn, wide, monkeypatch):
    monkeypatch.setattr(CH, "choose_wide", lambda specs, bn: wide and bn == CH.PAIR)
    rng = np.random.default_rng(0)
    specs = [_spec(L, m0, n0, formulation) for L, m0, n0 in shapes]
    xs = []
    for s in specs:
        x = rng.standard_normal((s.L, s.m0, s.n0))
        xs.append(x / np.linalg.norm(x, axis=(1, 2), keepdims=True))
    for s, x, out in zip(specs, xs, _interpret(specs, bn, xs)):
        for b in range(s.L):
            want = NS.direct_newton_schulz(torch.from_numpy(x[b]).double(), coefficients=s.coefs, eps=0.0,
                                           compute_dtype=torch.float64).numpy()
            # fp32 normalisation in the oracle, fp64 products on both sides
            assert np.abs(out[b] - want).max() < 1e-4 * np.abs(want).max()


def test_restart_variants_and_scale_factors():
    rng = np.random.default_rng(1)
    for restarts in ((), (1,), (2, 4), (0, 3)):
        s = _spec(1, 64, 136, restarts=restarts, h=0.25)
        x = rng.standard_normal((1, 64, 136))
        x /= np.linalg.norm(x)
        out = _interpret([s], 64, [x * 4.0])[0]
        want = NS.direct_newton_schulz(torch.from_numpy(x[0]).double(), coefficients=COEFS, eps=0.0,
                                       compute_dtype=torch.float64).numpy()
        assert np.abs(out[0] - want).max() < 1e-4 * np.abs(want).max()


def test_limits_of_a_plan():
    assert CH.fits([_spec(1, 128, 128)])
    assert not CH.fits([_spec(1, 128, 100)])                       # pitches are multiples of eight
    assert not CH.fits([_spec(0, 128, 128)])
    assert not CH.fits([_spec(1, 128, 128, coefs=COEFS * 20)])     # too many products
    assert not CH.fits([_spec(1, 128, 128)] * 17)
    # the largest batch that a Muon step makes is a plan
    from dmuon_b200.ops import ns_sm100
    for m, n in ((4096, 4096), (4096, 14336), (14336, 4096), (1032, 1160)):
        assert CH.possible((_spec(ns_sm100.max_batch(m, n), m, n),))
    # every tensor map is a kernel parameter: sixteen groups of the longest form that sixteen groups can have fit, more
    # operands than MAX_MAPS do not
    short = [_spec(1, 64 + 8 * i, 1024, coefs=COEFS[:1], restarts=()) for i in range(16)]
    maps = [sum(CH._map_count(s, bn) for s in short) for bn in (64, 128, 256)]
    assert CH.fits(short) and max(maps) <= CH.MAX_MAPS
    for L, m, n in ((1, 128, 14336), (1, 1152, 4304), (8, 256, 256), (1, 128, 128)):
        spl, per = CH.gram_splits(_spec(L, m, n), 128, CH.sym_tiles([_spec(L, m, n)], 128))
        kb = -(-n // 64)
        assert spl * per >= kb and (spl - 1) * per < kb and 1 <= spl <= 16


def test_tensor_maps_are_counted(monkeypatch):
    s = _spec(1, 128, 128)
    ops, _ = CH.build_entries([s], CH.choose_bn([s]))
    used = {m for _, pr, _, _, is_sum in ops if not is_sum for m in CH._operands(pr, CH.choose_bn([s]))}
    assert len(used) == CH._map_count(s, CH.choose_bn([s]))
    monkeypatch.setattr(CH, "MAX_MAPS", len(used) - 1)
    assert not CH.fits([s])


class _Memory:
    """Stands for an arena or a program: only who holds which."""

    def __init__(self, *args):
        self.args, self.captured, self.lists = args, False, self
        self.specs = args[0] if isinstance(args[0], tuple) else ()
        self.nbytes = CH.plan_bytes(self.specs) if self.specs else args[0]
        self.buf = self

    def numel(self):
        return self.nbytes

    def record_stream(self, stream):
        pass


@pytest.fixture
def streams(monkeypatch):
    """``plan_for`` without a device: the current stream and whether it captures are set by the test."""
    now = {"stream": 1, "capturing": False}
    monkeypatch.setattr(CH, "Program", _Memory)
    monkeypatch.setattr(CH, "Arena", _Memory)
    monkeypatch.setattr(CH, "Plan", lambda program, arena: type("P", (), dict(program=program, arena=arena)))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: now["capturing"])
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: now["stream"])
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: now["stream"], raising=False)
    for pool in ("_programs", "_plans", "_arenas"):
        monkeypatch.setattr(CH, pool, type(getattr(CH, pool))())
    return now


def test_captured_calls_have_work_memory_of_their_own(streams):
    dev = torch.device("cuda", 0)
    small, large = [_spec(1, 64, 128)], [_spec(1, 256, 512)]
    eager = CH.plan_for(small, dev)
    assert CH.plan_for(small, dev) is eager
    CH.plan_for(large, dev)                       # the arena grows: the smaller shape's plan goes with it
    streams.update(stream=7, capturing=True)
    first, second = CH.plan_for(small, dev), CH.plan_for(small, dev)
    streams["capturing"] = False
    plans = [first, second]
    for s in (1, 7):
        streams["stream"] = s
        plans += [CH.plan_for(large, dev), CH.plan_for(small, dev)]
    assert first.program is second.program is eager.program is plans[3].program is plans[5].program
    # two plans of one stream share its arena; nothing else shares anything
    assert plans[2].arena is plans[3].arena and plans[4].arena is plans[5].arena
    assert len({id(p.arena) for p in plans}) == 4
    assert not {id(p.arena) for p in (first, second)} & {id(a) for a in CH._arenas.values()}
    # the lists a graph names stay, whatever is given back or replaced
    CH.release()
    assert list(CH._programs.values()) == [first.program] and not CH._plans and not CH._arenas
    for i in range(CH.MAX_PLANS + 8):
        CH.plan_for([_spec(1, 64, 8 * (i + 20))], dev)
    assert len(CH._programs) <= CH.MAX_PLANS and first.program in CH._programs.values()
    assert len(CH._plans) <= CH.MAX_PLANS


def test_capture_without_an_earlier_call_has_no_plan(streams):
    streams["capturing"] = True
    assert CH.plan_for([_spec(1, 64, 128)], torch.device("cuda", 0)) is None
    assert not CH._programs


def test_jobs_whose_results_are_sent_have_launches_of_their_own(monkeypatch):
    """... and their callback comes before the next launch; the others share one."""
    import contextlib

    from dmuon_b200.ops import ns_sm100

    def job(m, n, apart):
        options = dict(coefs=COEFS, restarts=(2,), formulation="gram", compute_dtype=None, peer=None)
        return ns_sm100.UpdateJob([torch.zeros(m, n)], [torch.zeros(m, n)], [torch.zeros(m, n)], options, apart=apart)

    jobs = [job(64, 64, False), job(64, 128, True), job(64, 192, True), job(64, 256, False), job(64, 320, False)]
    events = []
    plan = type("P", (), dict(lock=contextlib.nullcontext()))
    monkeypatch.setattr(CH, "plan_for", lambda specs, device: plan)
    monkeypatch.setattr(ns_sm100, "_muon_update_chain",
                        lambda plan, part: events.append(["launch"] + [[x is j for x in jobs].index(True) for j in part]))
    ns_sm100.muon_update_groups(jobs, lambda i, wrote: events.append(i))
    assert events == [["launch", 0], 0, ["launch", 1], 1, ["launch", 2], 2, ["launch", 3, 4], 3, 4]


def test_work_memory_of_all_streams_is_bounded(streams):
    dev, spec = torch.device("cuda", 0), [_spec(8, 4096, 4096)]          # some 2.1 GB
    one = CH.plan_bytes(spec)
    for s in range(1, 8):
        streams["stream"] = s
        plan = CH.plan_for(spec, dev)
        assert CH._arenas[(0, s)] is plan.arena
        assert sum(a.numel() for a in CH._arenas.values()) <= CH.MAX_ARENA_BYTES
        assert len(CH._arenas) == min(s, CH.MAX_ARENA_BYTES // one)
        assert {k[1] for k in CH._plans} == set(CH._arenas)
    for s in range(20, 40):
        streams["stream"] = s
        CH.plan_for([_spec(1, 64, 128)], dev)
    assert len(CH._arenas) == CH.MAX_ARENAS

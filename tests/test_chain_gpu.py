"""One-launch Newton-Schulz (``csrc/chain_sm100.cu``) against 64-bit math (needs a B200)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("formulation", ["gram", "direct"])
@pytest.mark.parametrize("L,m0,n0,dt", [
    (1, 8, 64, torch.float32),            # far below one tile
    (1, 128, 128, torch.bfloat16),        # exactly one row of tiles
    (2, 136, 1040, torch.float32),        # remainders in every dimension, Gram split over K
    (1, 1152, 4304, torch.bfloat16),      # no multiple of a tile, full-width tiles, split
    (1, 4096, 200, torch.float32),        # tall: MN-major operands, split
    (1, 520, 520, torch.float32),         # full-width and half-width remainders of the mirror
    (5, 256, 256, torch.bfloat16),        # batch, several tickets per CTA
    (12, 1032, 1160, torch.bfloat16),     # CTA pairs, remainders in every dimension
    (450, 136, 520, torch.bfloat16),      # two tiles an entry in the last product, K of three and nine k-blocks
    (48, 1288, 1160, torch.float32),      # two tiles an entry, tall, K of 19 k-blocks: skewed head, middle and tail
    (75, 264, 128, torch.float32),        # CTA pairs, MN-major operands, K below one trip of the stage ring
])
def test_chain_matches_64_bit_iteration(L, m0, n0, dt, formulation, monkeypatch):
    from dmuon_b200.ops import chain as CH
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    torch.manual_seed(m0 + n0)
    coefs = list(NS.DEFAULT_COEFFICIENTS)
    restarts = [2] if formulation == "gram" else []
    X = (torch.randn(L, m0, n0, device=_dev()) * 1e-3).to(dt)
    for _ in range(3):                    # the kernel clears its counters for the next call
        out = ns_sm100.newton_schulz_batched(X, coefs, restarts, 1e-7, formulation)
    torch.cuda.synchronize()
    G.check_status(_dev())
    assert any(k[0][0][0].m0 == m0 and k[0][0][0].formulation == formulation for k in CH._plans)
    # the same products as one launch each: same operand roundings, 32-bit sums in the same order (another one where
    # a Gram product is split over K), so the two differ by what one changed rounding grows to in five steps
    monkeypatch.setattr(ns_sm100, "_chain_pays", lambda specs: False)
    alone = ns_sm100.newton_schulz_batched(X, coefs, restarts, 1e-7, formulation)
    torch.cuda.synchronize()
    G.check_status(_dev())
    for i in sorted({0, 1, L // 2, L - 1} & set(range(L))):
        exact = NS.direct_newton_schulz(X[i].double(), coefficients=coefs, compute_dtype=torch.float64)
        limit = 1.25 * _rel(alone[i], exact) + (2e-3 if formulation == "gram" else 8e-3)
        assert _rel(out[i], exact) < limit


def test_grouped_update_of_several_shapes_matches_fp32_math():
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    dev = _dev()
    torch.manual_seed(4)
    shapes = [(3, 256, 256), (2, 1024, 256), (2, 136, 512)]
    coefs, restarts, lr, wd, mu = list(NS.DEFAULT_COEFFICIENTS), [2], 0.02, 0.1, 0.9
    moms = [[torch.zeros(m, n, device=dev) for _ in range(L)] for L, m, n in shapes]
    masters = [[torch.randn(m, n, device=dev) * 0.02 for _ in range(L)] for L, m, n in shapes]
    pubs = [[torch.zeros(m, n, device=dev, dtype=torch.bfloat16) for _ in range(L)] for L, m, n in shapes]
    for step, mag in enumerate([1e-3, 5e-3, 2.5e-4]):
        grads = [[(torch.randn(m, n, device=dev) * mag).bfloat16() for _ in range(L)] for L, m, n in shapes]
        m_prev = [[x.clone() for x in g] for g in moms]
        w_prev = [[x.clone() for x in g] for g in masters]
        jobs = []
        for g, (L, m, n) in enumerate(shapes):
            options = dict(mu=mu, nesterov=True, coefs=coefs, restarts=restarts, formulation="gram", lr=lr,
                           weight_decay=wd, update_scale=0.2 * math.sqrt(max(m, n)), compute_dtype=None, gscale=None,
                           peer=None)
            jobs.append(ns_sm100.UpdateJob(grads[g], moms[g], masters[g], options, publish=pubs[g] if g else None))
        issued = {}
        ns_sm100.muon_update_groups(jobs, issued.__setitem__)
        torch.cuda.synchronize()
        G.check_status(dev)
        assert issued == {0: False, 1: True, 2: True}
        for g, (L, m, n) in enumerate(shapes):
            scale = 0.2 * math.sqrt(max(m, n))
            for i in range(L):
                buf = mu * m_prev[g][i] + grads[g][i].float()
                u = grads[g][i].float() + mu * buf
                o = NS.gram_newton_schulz(u, coefficients=coefs, restart_iterations=restarts, deterministic=True,
                                          compute_dtype=torch.float32)
                ref = w_prev[g][i] * (1 - lr * wd) - lr * scale * o
                assert torch.allclose(moms[g][i], buf, atol=1e-6), (step, g)
                # The step itself, relative to its 2-norm: a correction factor that is off by a few percent shows.  fp16
                # products: 0.005 seen where the matrix is well conditioned.  Square random ones: a Gram matrix in fp16
                # does not resolve singular values below sqrt(2^-11) = 0.022 of the largest (2 sqrt(n)); the k-th smallest
                # of n lies at k pi / (2 sqrt(n)), so that is a share of 0.022 * 4 / pi = 0.028 of the directions, and
                # with those wholly off the error is sqrt(0.028) = 0.17
                step_ref = ref - w_prev[g][i] * (1 - lr * wd)
                off = (masters[g][i] - ref).norm() / step_ref.norm()
                assert off < (0.17 if m == n else 1.5e-2), (step, g, off.item())
                if g:
                    assert torch.equal(pubs[g][i], masters[g][i].bfloat16())


def test_chain_on_two_streams_at_once():
    """Plans are per stream: calls of one shape on two streams do not share buffers."""
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    coefs, dev = list(NS.DEFAULT_COEFFICIENTS), _dev()
    torch.manual_seed(5)
    X = [torch.randn(1, 256, 640, device=dev) for _ in range(2)]
    want = [ns_sm100.newton_schulz_batched(x, coefs, [2]) for x in X]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(dev) for _ in X], []
    for _ in range(8):
        for x, s in zip(X, streams):
            with torch.cuda.stream(s):
                got.append(ns_sm100.newton_schulz_batched(x, coefs, [2]))
    torch.cuda.synchronize()
    G.check_status(dev)
    for k, o in enumerate(got):
        # the norm is an atomic sum: its last bit, amplified by five fp16 steps
        assert _rel(o, want[k % 2].double()) < 2e-2


def test_plans_that_follow_each_other_on_recycled_memory():
    """Arenas grow, plans go and others take their addresses: every launch uses its own tensor maps."""
    from dmuon_b200.ops import chain as CH
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    coefs, dev = list(NS.DEFAULT_COEFFICIENTS), _dev()
    torch.manual_seed(8)
    shapes = [(64, 136), (72, 200), (256, 64), (256, 512), (512, 1032), (1032, 264), (1024, 2048), (64, 136), (256, 512)]
    for turn in range(3):
        for m, n in shapes:
            x = torch.randn(1, m, n, device=dev)
            exact = NS.direct_newton_schulz(x[0].double(), coefficients=coefs, compute_dtype=torch.float64)
            # fp16 products of five steps on matrices that are not square (well conditioned): 0.0045 seen
            assert _rel(ns_sm100.newton_schulz_batched(x, coefs, [2])[0], exact) < 2e-2, (turn, m, n)
        CH.release()
    torch.cuda.synchronize()
    G.check_status(dev)


def _graph_of(fn, x):
    static_in = x.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        static_out = fn(static_in)
    return graph, static_in, static_out


def test_shapes_called_in_ascending_order_can_be_captured():
    """Work memory that grew for a larger shape does not take a smaller one's plan from a later capture."""
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS
    from dmuon_b200.optim import ns_graph

    coefs, dev = list(NS.DEFAULT_COEFFICIENTS), _dev()
    torch.manual_seed(9)

    def fn(x):
        return ns_sm100.newton_schulz_batched(x, coefs, [2])

    # sizes of no other test: the separate launches have no tile lists of them either.  bf16: the norm's last bit,
    # which is an atomic sum, does not show
    xs = [torch.randn(1, m, n, device=dev).bfloat16() for m, n in ((264, 1096), (968, 2120), (1416, 2664))]
    want = [fn(x) for x in xs]
    graphs = [_graph_of(fn, x) for x in xs]
    cache = ns_graph.NSGraphCache()
    for turn in range(3):
        for x, w, (graph, static_in, static_out) in zip(xs, want, graphs):
            static_in.copy_(x)
            graph.replay()
            assert _rel(static_out, w.double()) < 1e-2
            assert _rel(cache.run(tuple(x.shape), fn, x), w.double()) < 1e-2
    torch.cuda.synchronize()
    G.check_status(dev)
    assert cache.stats() == dict(keys=3, captures=3, replays=6, failed=0)


def test_replays_beside_eager_calls_on_other_streams():
    """A graph's work memory and counters are its own: two graphs of one shape and eager calls of this and
    another shape run at once on four streams."""
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    coefs, dev = list(NS.DEFAULT_COEFFICIENTS), _dev()
    torch.manual_seed(10)

    def fn(x):
        return ns_sm100.newton_schulz_batched(x, coefs, [2])

    a = [torch.randn(1, 520, 1160, device=dev).bfloat16() for _ in range(3)]
    b = torch.randn(1, 776, 1288, device=dev).bfloat16()
    want, want_b = [fn(x) for x in a], fn(b)
    graphs = [_graph_of(fn, x) for x in a[:2]]
    streams = [torch.cuda.Stream(dev) for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for _ in range(10):
        for k, (graph, _, static_out) in enumerate(graphs):
            with torch.cuda.stream(streams[k]):
                graph.replay()
                got.append((static_out.clone(), want[k]))
        with torch.cuda.stream(streams[2]):
            got.append((fn(b), want_b))
            got.append((fn(a[2]), want[2]))
        got.append((fn(b), want_b))
        got.append((fn(a[2]), want[2]))
    torch.cuda.synchronize()
    G.check_status(dev)
    for out, w in got:
        assert _rel(out, w.double()) < 1e-2


class _LocalPeer:
    """The gradients of a batch as the peer plane hands them over, all on this GPU."""

    def __init__(self, grads):
        self.keep = torch.cat([g.reshape(-1) for g in grads])
        self.peer_bases, self.grad_dtype, self.scale = [self.keep.data_ptr()], self.keep.dtype, 1.0
        self.numels = [g.numel() for g in grads]
        self.offsets = [sum(self.numels[:i]) for i in range(len(grads))]
        self.ready_flags, self.ready_want, self.status = None, 0, None


class _LocalShards:
    """The gradients of a batch as tensor-parallel shards (halves of the rows), all on this GPU."""

    def __init__(self, grads):
        self.shards = [[s.contiguous() for s in g.chunk(2)] for g in grads]

    def launch_prologue(self, moms, xs, slots, sumsq, **kw):
        from dmuon_b200.ops import tp_peer as TP

        jobs = []
        for i, pair in enumerate(self.shards):
            row = 0
            for s in pair:
                jobs.append(TP.ShardJob(i, s.data_ptr(), s.shape[0], s.shape[1], row * s.shape[1], s.shape[1]))
                row += s.shape[0]
        TP.gather_prologue(jobs, self.shards[0][0].dtype, moms, xs, slots, sumsq, **kw)


@pytest.mark.parametrize("form", ["chain", "launches", "peer", "shards"])
@pytest.mark.parametrize("mom_dtype", [torch.float32, torch.bfloat16])
def test_update_after_zero_and_jumping_gradients(form, mom_dtype, monkeypatch):
    """The factor that an fp16 operand is stored with is last step's; steps after which it does not do."""
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    if form != "chain":
        monkeypatch.setattr(ns_sm100, "_chain_pays", lambda specs: False)
    dev = _dev()
    torch.manual_seed(12)
    shapes = [(3, 264, 1024), (2, 1032, 256)]
    coefs, restarts, lr, wd, mu = list(NS.DEFAULT_COEFFICIENTS), [2], 0.02, 0.1, 0.9
    moms = [[torch.zeros(m, n, device=dev, dtype=mom_dtype) for _ in range(L)] for L, m, n in shapes]
    masters = [[torch.randn(m, n, device=dev) * 0.02 for _ in range(L)] for L, m, n in shapes]
    # magnitudes of the gradients, whether the momentum starts from zero: no gradient at all, a norm 1e5 times as large,
    # one 1e10 times smaller, 50 times either way (inside the range of a stored factor), zero again
    for step, (mag, zero) in enumerate([(0.0, False), (1e-3, False), (1e2, False), (1e-8, True), (5e-7, True),
                                        (1e-8, True), (0.0, True), (1e-2, False), (1e-2, False)]):
        grads = [[(torch.randn(m, n, device=dev) * mag).bfloat16() for _ in range(L)] for L, m, n in shapes]
        if step == 4:
            grads[0][1].zero_()               # one matrix of a batch
        if zero:
            for x in (*moms[0], *moms[1]):
                x.zero_()
        m_prev = [[x.clone() for x in g] for g in moms]
        w_prev = [[x.clone() for x in g] for g in masters]
        jobs = []
        for g, (L, m, n) in enumerate(shapes):
            peer = {"peer": _LocalPeer, "shards": _LocalShards}.get(form, lambda grads: None)(grads[g])
            options = dict(mu=mu, nesterov=True, coefs=coefs, restarts=restarts, formulation="gram", lr=lr,
                           weight_decay=wd, update_scale=0.2 * math.sqrt(max(m, n)), compute_dtype=None, gscale=None,
                           peer=peer)
            jobs.append(ns_sm100.UpdateJob(grads[g] if peer is None else None, moms[g], masters[g], options))
        ns_sm100.muon_update_groups(jobs, lambda i, wrote: None)
        torch.cuda.synchronize()
        G.check_status(dev)
        for g, (L, m, n) in enumerate(shapes):
            for i in range(L):
                buf = (mu * m_prev[g][i].float() + grads[g][i].float()).to(mom_dtype).float()
                u = grads[g][i].float() + mu * buf
                o = NS.gram_newton_schulz(u, coefficients=coefs, restart_iterations=restarts, deterministic=True,
                                          compute_dtype=torch.float32)
                delta = masters[g][i] - w_prev[g][i] * (1 - lr * wd)
                want = -lr * 0.2 * math.sqrt(max(m, n)) * o
                # one rounding here, two in the kernel's fused form
                ulp = 1e-2 if mom_dtype == torch.bfloat16 else 1e-6
                assert torch.allclose(moms[g][i].float(), buf, rtol=ulp, atol=ulp * float(buf.abs().max()))
                # fp16 products on well conditioned matrices, 0.005 seen; a result of zeros leaves the rounding of the
                # weight itself (6e-8 of 0.02)
                assert (delta - want).norm() < 1.5e-2 * want.norm() + 1e-8 * math.sqrt(m * n), (step, g, i)


def test_update_with_changing_participation():
    """A matrix without a gradient in a step: the others' stored factors serve on, all results stay right."""
    from dmuon_b200.ops import chain as CH
    from dmuon_b200.ops import gemm as G
    from dmuon_b200.ops import ns_sm100
    from dmuon_b200.optim import newton_schulz as NS

    dev = _dev()
    torch.manual_seed(13)
    shapes = [(4, 136, 520), (2, 264, 1024), (2, 520, 136)]
    coefs, restarts, lr, mu = list(NS.DEFAULT_COEFFICIENTS), [2], 0.02, 0.9
    moms = [[torch.zeros(m, n, device=dev) for _ in range(L)] for L, m, n in shapes]
    masters = [[torch.randn(m, n, device=dev) * 0.02 for _ in range(L)] for L, m, n in shapes]
    CH.release()
    for step, idle in enumerate([(), (2,), (), (0, 3), (2,), ()]):
        here = [[i for i in range(L) if g or i not in idle] for g, (L, _, _) in enumerate(shapes)]
        grads = [[(torch.randn(m, n, device=dev) * 1e-3).bfloat16() for _ in range(L)] for L, m, n in shapes]
        m_prev = [[x.clone() for x in g] for g in moms]
        w_prev = [[x.clone() for x in g] for g in masters]
        jobs = []
        for g, (L, m, n) in enumerate(shapes):
            options = dict(mu=mu, nesterov=True, coefs=coefs, restarts=restarts, formulation="gram", lr=lr,
                           weight_decay=0.0, update_scale=1.0, compute_dtype=None, gscale=None, peer=None)
            pick = lambda ts: [ts[i] for i in here[g]]
            jobs.append(ns_sm100.UpdateJob(pick(grads[g]), pick(moms[g]), pick(masters[g]), options))
        ns_sm100.muon_update_groups(jobs, lambda i, wrote: None)
        torch.cuda.synchronize()
        G.check_status(dev)
        plan = next(reversed(CH._plans.values()))
        assert plan.n_matrices == sum(map(len, here))
        if step:
            assert not plan.again[len(here[0]):].any()
        for g, (L, m, n) in enumerate(shapes):
            for i in range(L):
                if i not in here[g]:
                    assert torch.equal(masters[g][i], w_prev[g][i]) and torch.equal(moms[g][i], m_prev[g][i])
                    continue
                u = grads[g][i].float() + mu * moms[g][i]
                o = NS.gram_newton_schulz(u, coefficients=coefs, restart_iterations=restarts, deterministic=True,
                                          compute_dtype=torch.float32)
                # as above: fp16 products on well conditioned matrices
                assert _rel(masters[g][i] - w_prev[g][i], -lr * o.double()) < 1.5e-2, (step, g, i)

"""hh_solve_source_multi past the plans (16) and chunks (64) whose table travels in the kernel's arguments: the
table is copied to device memory, or, in a stream capture, the line solve goes plan by plan.  The fields of every
plan are bitwise its own solves."""
import pytest

import hackathon_b200 as hh

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _problem(stream, dim, n, order, nplans, counts):
    """A context on `stream`, plans at different k, one batch for them and the solo solves of its fields."""
    ctx = hh.Context(0, stream.cuda_stream)
    plans = [hh.Plan.helmholtz(ctx, dim, n, order, 2.0 + 1.25 * i + (0.5j if i % 5 == 4 else 0)) for i in range(nplans)]
    g = torch.Generator(device="cuda").manual_seed(n + nplans)
    f = torch.view_as_complex(torch.randn((sum(counts),) + (n,) * dim + (2,), dtype=torch.float64, device="cuda", generator=g))
    solo, off = torch.empty_like(f), 0
    torch.cuda.synchronize()
    for p, c in zip(plans, counts):
        p.solve_source(f[off:off + c], solo[off:off + c], c)
        off += c
    ctx.synchronize()
    return ctx, plans, f, solo


# 16 plans and 64 chunks (of one right-hand side each, at short lines) are the last that fit the arguments
SHAPES = [(2, 63, 6, 16, [1] * 16), (2, 63, 6, 17, [1] * 17), (2, 255, 4, 40, [2, 1] * 20), (3, 31, 6, 17, [1] * 17),
          (2, 63, 2, 2, [32, 32]), (2, 63, 2, 2, [33, 32]), (2, 255, 4, 17, [16] * 17)]  # (the last: a padded workspace)


@pytest.mark.parametrize("dim,n,order,nplans,counts", SHAPES)
def test_multi_in_a_capture_equals_solo_solves(dim, n, order, nplans, counts):
    """A replay of the captured solve gives the bits of the solo solves, on inputs written after the capture."""
    stream = torch.cuda.Stream()
    ctx, plans, f, solo = _problem(stream, dim, n, order, nplans, counts)
    src, u = torch.zeros_like(f), torch.empty_like(f)
    torch.cuda.synchronize()
    hh.solve_source_multi(plans, counts, src, u)  # buffers grown on demand are there before the capture
    ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        hh.solve_source_multi(plans, counts, src, u)
    src.copy_(f)
    for _ in range(2):
        u.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(u, solo)
    del graph
    ctx.close()


@pytest.mark.parametrize("dim,n,order,nplans,counts", SHAPES)
def test_multi_equals_solo_solves(dim, n, order, nplans, counts):
    """One call and one line-solve launch (the table in the arguments or in device memory), the solo solves' bits."""
    ctx, plans, f, solo = _problem(torch.cuda.Stream(), dim, n, order, nplans, counts)
    u = torch.full_like(f, float("nan"))
    torch.cuda.synchronize()
    before = ctx.launches
    hh.solve_source_multi(plans, counts, f, u)
    ctx.synchronize()
    assert ctx.launches - before == (3 if dim == 2 else 5)
    assert torch.equal(u, solo)
    ctx.close()


def test_request_loop_merges_more_plans_than_the_arguments_hold(ctx):
    """Sixty requests of one shape, each at its own k, queued while the loop sets up: it merges batches of more than
    16 plans, and every request gets its solo solve."""
    hh.tune_cache_clear()
    n = 63
    ks = [1.0 + 0.6 * i for i in range(60)]
    g = torch.Generator(device="cuda").manual_seed(8)
    f = torch.view_as_complex(torch.randn((60, n, n, 2), dtype=torch.float64, device="cuda", generator=g))
    u = torch.empty_like(f)
    torch.cuda.synchronize()
    srv = hh.Server(0, hbm_budget=4 << 30, streams=2)
    ids = [srv.submit(2, n, 6, k, 1, f[i], u[i], on_device=True) for i, k in enumerate(ks)]
    infos = [srv.wait(i) for i in ids]
    srv.close()
    assert max(i["batch_rhs"] for i in infos) > 16
    for i, k in enumerate(ks):
        plan = hh.Plan.helmholtz(ctx, 2, n, 6, k)
        solo = torch.empty_like(f[i])
        plan.solve_source(f[i], solo, 1)
        ctx.synchronize()
        assert torch.equal(u[i], solo)
        plan.close()


def test_first_multi_solve_may_be_captured():
    """Three plans need no device table, so a context's very first multi solve allocates nothing."""
    stream = torch.cuda.Stream()
    ctx, plans, f, solo = _problem(stream, 2, 127, 4, 3, [2, 1, 2])
    u = torch.empty_like(f)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        hh.solve_source_multi(plans, [2, 1, 2], f, u)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(u, solo)
    del graph
    ctx.close()

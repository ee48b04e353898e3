"""Kernels of a solve start while the one before drains, and set up from tables and factors before they wait: work
queued back to back -- plans made, used and destroyed between other solves, several contexts on one stream, a context
moved between streams -- gives the bits of the same calls with a wait after each."""
import pytest

import hackathon_b200 as hh

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _field(dim, n, batch, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn((batch,) + (n,) * dim + (2,), dtype=torch.float64, device="cuda", generator=g))


KINDS = [(2, 63, 6), (2, 100, 4), (3, 31, 4), (2, 255, 6), (3, 20, 6), (2, 47, 2)]


def test_plans_made_and_destroyed_between_queued_solves():
    """A kept plan's solves run on through the set-up, one solve and the end of other plans; each new plan of a round
    has a length of its own (new tables) or the memory of the plan destroyed before it."""
    def run(wait):
        stream = torch.cuda.Stream()
        ctx = hh.Context(0, stream.cuda_stream)
        kept = hh.Plan.helmholtz(ctx, 2, 127, 6, 20.0)
        x = _field(2, 127, 3, 1)
        fields = [_field(d, n, 2, 10 + i) for i, (d, n, _) in enumerate(KINDS)]
        torch.cuda.synchronize()
        for round_ in range(3):
            for (d, n, o), f in zip(KINDS, fields):
                for _ in range(3):
                    kept.solve_source(x, x, 3)
                    if wait:
                        ctx.synchronize()
                p = hh.Plan.helmholtz(ctx, d, n, o, 3.0 + round_)
                p.solve_source(f, f, 2)
                if wait:
                    ctx.synchronize()
                kept.solve_source(x, x, 3)
                p.close()
                if wait:
                    ctx.synchronize()
            x.mul_(1e6)  # (a solve shrinks the field)
            torch.cuda.synchronize()
        ctx.synchronize()
        out = [x] + fields
        ctx.close()
        return out

    for a, b in zip(run(False), run(True)):
        assert torch.isfinite(torch.view_as_real(a)).all() and torch.equal(a, b)


@pytest.mark.parametrize("dim,n,order", KINDS)
def test_contexts_on_one_stream(dim, n, order):
    """Three contexts on one stream, each solving what the one before left."""
    def run(wait):
        stream = torch.cuda.Stream()
        ctxs = [hh.Context(0, stream.cuda_stream) for _ in range(3)]
        x = _field(dim, n, 2, n)
        torch.cuda.synchronize()
        plans = [hh.Plan.helmholtz(c, dim, n, order, 2.0 + i + (0.5j if i == 2 else 0)) for i, c in enumerate(ctxs)]
        for _ in range(4):
            for c, p in zip(ctxs, plans):
                p.solve_source(x, x, 2)
                if wait:
                    c.synchronize()
        torch.cuda.synchronize()
        for c in ctxs:
            c.close()
        return x

    assert torch.equal(run(False), run(True))


def test_context_moved_between_streams():
    """The context's stream changes between solves, each stream waiting for the one before by an event."""
    def run(wait):
        streams = [torch.cuda.Stream() for _ in range(3)]
        ctx = hh.Context(0, streams[0].cuda_stream)
        x, y = _field(2, 100, 2, 3), _field(3, 31, 2, 4)
        torch.cuda.synchronize()
        p = hh.Plan.helmholtz(ctx, 2, 100, 6, 9.0)
        for i in range(12):
            ctx.set_stream(streams[i % 3].cuda_stream)
            p.solve_source(x, x, 2)
            q = hh.Plan.helmholtz(ctx, 3, 31, 6, 2.0 + i % 2)
            q.solve_source(y, y, 2)
            streams[(i + 1) % 3].wait_stream(streams[i % 3])
            q.close()
            if wait:
                ctx.synchronize()
        torch.cuda.synchronize()
        ctx.close()
        return x, y

    for a, b in zip(run(False), run(True)):
        assert torch.equal(a, b)

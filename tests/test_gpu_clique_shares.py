"""A 4-clique split over ranks.  Which cliques a rank counts depends on the
relation and the number of ranks alone: a rank whose card has no memory for the
hit masks counts the same ones by the plan without masks, so the shares still add
up.  And one vertex next to most others is dealt out, it does not leave its work
to one rank.  The shares run one after another on this GPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub(d, extra, core, kind="up", seed=3, hubs=1):
    """`hubs` vertices, each next to d others; `extra` random edges among those, and
    a clique of `core`."""
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, d, extra) + hubs, rng.integers(0, d, extra) + hubs
    ca, cb = np.triu_indices(core, 1)
    ids = np.sort(rng.choice(np.arange(hubs, d + hubs), core, replace=False))
    u = np.concatenate([np.repeat(np.arange(hubs), d), np.minimum(a, b), ids[ca]])
    v = np.concatenate([np.tile(np.arange(hubs, d + hubs), hubs), np.maximum(a, b), ids[cb]])
    keep = u != v
    u, v = u[keep].astype(np.uint32), v[keep].astype(np.uint32)
    if kind == "down":
        u, v = v, u
    if kind == "sym":
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    return u, v


class _FillTo:
    """Leaves `free` bytes of the device's memory to the engine."""

    def __init__(self, ctx, free):
        self.ctx, self.free = ctx, free

    def __enter__(self):
        import torch
        self.ctx.reserve(0)
        torch.cuda.empty_cache()
        self.hold = torch.empty(torch.cuda.mem_get_info()[0] - self.free, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        del self.hold
        torch.cuda.empty_cache()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
def test_a_rank_without_memory_counts_the_same_share(eh, ctx, oracle, kind):
    # masks of 56 * 40,000^2 / 64 words are 5.6 GB, on a rank of three a third of
    # the hubs' ones 1.9; the plan without them takes 0.9 GB
    u, v = _hub(40_000, 20_000, 60, kind, hubs=56)
    t = eh.Trie(u, v, ctx=ctx)
    want = oracle.Trie(u, v).clique4()
    assert want >= 60 * 59 * 58 * 57 // 24
    assert t.count("clique4") == want
    shares = [t.count("clique4", shard=(r, 3)) for r in range(3)]
    assert sum(shares) == want
    for r in range(3):
        with _FillTo(ctx, 1500 << 20):
            assert t.count("clique4", shard=(r, 3)) == shares[r], r
    t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("d,extra,core", [(33, 60, 12), (100, 2000, 20), (3000, 20000, 90), (9000, 100, 300)])
def test_shares_of_a_hub(eh, oracle, kind, d, extra, core):
    u, v = _hub(d, extra, core, kind)
    t = eh.Trie(u, v)
    want = oracle.Trie(u, v).clique4()
    for world in (2, 3, 8, 37):
        assert sum(t.count("clique4", shard=(r, world)) for r in range(world)) == want, world
    t.free()


@pytest.mark.parametrize("kind", ["up", "down", "sym"])
@pytest.mark.parametrize("rows", [-40, 0, 40])
def test_shares_at_the_hub_rule(eh, oracle, kind, rows):
    """A part of d elements around the line where the rows fill a 1024th of its matrix."""
    d = 4400
    u, v = _hub(d, 4950 + rows, 30, kind)
    t = eh.Trie(u, v)
    want = oracle.Trie(u, v).clique4()
    for world in (2, 5):
        assert sum(t.count("clique4", shard=(r, world)) for r in range(world)) == want, world
    t.free()


def test_shares_of_a_star_are_even(eh):
    """2^16 vertices next to vertex 0 and few rows among them: no rank takes over
    half as long as the whole."""
    t = eh.Trie(*_hub(1 << 16, 1 << 18, 4))

    def ms(**kw):
        return min(t.count("clique4", stats=True, **kw)[1]["kernel_ms"] for _ in range(4))

    assert max(ms(shard=(r, 8)) for r in range(8)) < 0.5 * ms()
    t.free()


def test_shares_of_a_hub_are_even(eh):
    """R-MAT-15 by its own ids: vertex 0 meets a third of all vertices."""
    u, v = eh.gen_rmat(5, 15, 16 << 15)
    u, v = u.numpy(), v.numpy()
    u, v = np.minimum(u, v)[u != v], np.maximum(u, v)[u != v]
    t = eh.Trie(u, v)

    def ms(**kw):
        return min(t.count("clique4", stats=True, **kw)[1]["kernel_ms"] for _ in range(4))

    # the masks of the widest part are made on every rank, its rows are not repeated
    assert max(ms(shard=(r, 8)) for r in range(8)) < 0.5 * ms()
    t.free()

"""Multi-GPU plumbing for one COUNT query split across ranks.

Every rank holds the whole trie (0.3-1.3 GB at the benchmark sizes; HBM is
180 GB) and runs its share of the heaviest-first plan: item i of head entry b
where (b + i) % world == rank (of an item that a group of 8 or 16 neighbouring
entries share, the group's number in place of b); for the 4-clique of an up, down or symmetric
relation the cliques of the head entries a with a % world == rank, those of the
widest entries by eight rows (eh_exec_config.shard_index / shard_count).  The
only exchange is the final sum: one 8-byte all-reduce.  Counts are modulo 2^64
like the reference's signed long, so the sum is taken on int64 tensors and
read back as uint64 bit patterns.  The reference's own parallelism is the
same split over threads (par::for_range + par::reducer,
storage_engine/src/utils/parallel.cpp:42-79, utils/parallel.hpp:8-34).
"""
import torch

MASK64 = (1 << 64) - 1


def to_i64(u):
    """uint64 bit pattern -> int64 value with the same bits."""
    u &= MASK64
    return u - (1 << 64) if u >= (1 << 63) else u


def combine_counts(count, device="cpu", group=None):
    """Sum of every rank's partial count, modulo 2^64."""
    import torch.distributed as dist
    t = torch.tensor([to_i64(int(count))], dtype=torch.int64, device=device)
    if dist.is_available() and dist.is_initialized():
        dist.all_reduce(t, group=group)
    return int(t.item()) & MASK64


def max_over_ranks(x, device="cpu", group=None):
    import torch.distributed as dist
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    if dist.is_available() and dist.is_initialized():
        dist.all_reduce(t, op=dist.ReduceOp.MAX, group=group)
    return float(t.item())


def owned(n_items, rank, world, entry=0):
    """Indices i of the n_items items of a head entry that a rank runs:
    (entry + i) % world == rank, the device's rule."""
    return range((rank - entry) % world, n_items, world)

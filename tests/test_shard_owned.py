"""The host mirror of the rule that deals a head entry's work items to ranks."""
import pytest


@pytest.mark.parametrize("world", [1, 2, 3, 8])
def test_items_of_an_entry_are_dealt_from_its_number(world):
    from emptyheaded_b200 import shard
    for n in (0, 1, 5, 40):
        for entry in (0, 1, 7, 8, 1001):
            got = {i: r for r in range(world) for i in shard.owned(n, r, world, entry)}
            assert got == {i: (entry + i) % world for i in range(n)}

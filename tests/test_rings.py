"""The ring of ``project_split_kernel`` (landmark_b200/csrc/gnr_project_split.cu), every interleaving of its roles: two
groups of gather warps store pairs into six slots, one warp issues MMAs in order, the tensor pipe consumes them in order.
A slot's barriers are waited for by parity alone, so an order of the pairs is sound only if no interleaving lets a warp
store into a slot that is not consumed, or stops.  (CPU: a model of the protocol, with the kernel's order of pairs.)"""
import pytest

SLOTS, WARPS = 6, 2  # warps per group: two show everything that eight can (one ahead, one behind)


def _order(n_pairs, tiles, group, by_pairs):
    """The pairs a group's warps store, numbered through the tiles (``n * n_pairs + pi``)."""
    if by_pairs:
        return [n * n_pairs + pi for n in range(tiles) for pi in range((group + n * n_pairs) & 1, n_pairs, 2)]
    return [n * n_pairs + pi for n in range(group, tiles, 2) for pi in range(n_pairs)]


def _explore(n_pairs, tiles, by_pairs):
    total = n_pairs * tiles
    orders = [_order(n_pairs, tiles, w // WARPS, by_pairs) for w in range(2 * WARPS)]
    start = ((0,) * (2 * WARPS), (0,) * SLOTS, (0,) * SLOTS, 0, 0)  # positions, arrivals, full phases, issued, consumed
    seen, todo = {start}, [start]
    while todo:
        at, arrived, full, issued, consumed = todo.pop()
        after = []
        for w, order in enumerate(orders):
            if at[w] == len(order):
                continue
            q = order[at[w]]
            slot, use = q % SLOTS, q // SLOTS
            freed = max(0, (consumed - slot + SLOTS - 1) // SLOTS)  # completed phases of the slot's "empty" barrier
            if use > 0 and (freed & 1) == ((use - 1) & 1):
                continue  # the parity wait blocks
            if consumed < q - SLOTS + 1:
                return f"pair {q} stored while {consumed} are consumed"
            a, f = list(arrived), list(full)
            a[slot] += 1
            if a[slot] == WARPS:
                a[slot], f[slot] = 0, f[slot] + 1
            after.append((at[:w] + (at[w] + 1,) + at[w + 1:], tuple(a), tuple(f), issued, consumed))
        if issued < total and (full[issued % SLOTS] & 1) != (issued // SLOTS & 1):
            if full[issued % SLOTS] <= issued // SLOTS:
                return f"pair {issued} read before it is stored"
            after.append((at, arrived, full, issued + 1, consumed))
        if consumed < issued:
            after.append((at, arrived, full, issued, consumed + 1))
        if not after and consumed < total:
            return f"stops with {consumed} of {total} consumed"
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return "sound"


@pytest.mark.parametrize("n_pairs", range(1, 10))
def test_projection_ring_is_sound(n_pairs):
    by_pairs = n_pairs >= SLOTS  # the kernel's rule
    assert _explore(n_pairs, 4, by_pairs) == "sound"
    if by_pairs:  # (why the rule lies there: tile by tile, a group's parity wait can pass a use too early)
        assert "stored while" in _explore(n_pairs, 4, False)

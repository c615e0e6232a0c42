"""The neighbour-cell table has room for every cell's runs and no more, checked by a restatement of its kernel."""
import itertools
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "threebodymdalgorithms_b200" / "csrc" / "tbmd_internal.cuh"


def runs(dims, c):
    """Runs of consecutive ids >= c among the neighbours of cell c in a periodic grid."""
    at = c % dims[0], c // dims[0] % dims[1], c // (dims[0] * dims[1])
    off = [(0,) if d == 1 else (-1, 0, 1) for d in dims]
    ids = set()
    for d in itertools.product(*off):
        x, y, z = ((a + s) % n for a, s, n in zip(at, d, dims))
        ids.add((z * dims[1] + y) * dims[0] + x)
    ids = sorted(i for i in ids if i >= c)
    return 1 + sum(b != a + 1 for a, b in zip(ids, ids[1:]))


def test_room_for_every_cell():
    """An axis has one cell or at least three; from five on only the distance of the wrapped neighbour grows."""
    room = int(re.search(r"constexpr int NB_RUNS = (\d+);", SOURCE.read_text()).group(1))
    most = max(runs(dims, c) for dims in itertools.product([1, 3, 4, 5, 6, 7], repeat=3)
               for c in range(dims[0] * dims[1] * dims[2]))
    assert most == room

"""Host model of the warp form of compact_row (csrc/peel.cu): 32 lanes read an
entry each, vote on which stay, and write those to lower places of the same
arrays.  A vote orders no memory, and the ids that a lane reads do not feed it,
so without a warp synchronisation before the writes a lane may read its id
after another one has written there.  The model replays random schedules of
the reads and writes with the synchronisation that the source has."""
import os
import random
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tdtdecomposition_gb300", "csrc",
                   "peel.cu")


def _source_has_sync():
    """The warp form meets at a __syncwarp between the votes and the writes."""
    src = open(SRC).read()
    body = src[src.index("int compact_row("):]
    body = body[:body.index("\n}\n")]
    vote, write = body.index("__ballot_sync"), body.index("ids[to] =")
    return re.search(r"__syncwarp\(\)", body[vote:write]) is not None


def compact(ids, keep, sync, rng, lanes=32):
    out, n = list(ids), 0
    for t in range(0, len(ids), lanes):
        tile = range(t, min(t + lanes, len(ids)))
        kept = [i for i in tile if keep[i]]
        to = {i: n + k for k, i in enumerate(kept)}
        reads = [("read", i) for i in tile]
        rng.shuffle(reads)
        if sync:
            writes = [("write", i) for i in kept]
            rng.shuffle(writes)
            events = reads + writes
        else:  # a lane's write follows its own read, and nothing else
            events = [e for r in reads for e in [r] + ([("write", r[1])] if keep[r[1]] else [])]
        reg = {}
        for kind, i in events:
            if kind == "read":
                reg[i] = out[i]
            else:
                out[to[i]] = reg[i]
        n += len(kept)
    return out[:n]


def _schedules(sync):
    rng = random.Random(5)
    wrong = 0
    for _ in range(300):
        n = rng.randint(1, 200)
        ids = list(range(1000, 1000 + n))
        keep = [rng.random() < 0.7 for _ in ids]
        wrong += compact(ids, keep, sync, rng) != [x for x, k in zip(ids, keep) if k]
    return wrong


def test_rows_compact_in_order_under_any_schedule():
    assert _schedules(_source_has_sync()) == 0


def test_the_synchronisation_is_needed():
    assert _schedules(True) == 0 and _schedules(False) > 0

"""The producer / consumer protocol of the warp-specialised kernels (k_sc_ws
in ws.cuh, k_thermal_ws in thermal_ws.cuh), model-checked on the CPU.

The model follows the kernels' order of operations, one step at a time, and
runs it under random interleavings of one producer warp and three consumer
warps:

* producer: publish the descriptors (neighbour row, block id, ghost row) of
  blocks 0 and 1 and signal "ready"; then for each block j: publish block
  j+1's descriptors (j >= 1), wait until every consumer has released block
  j - B (B stage buffers), and issue block j's copies into buffer j % B (the
  "landed" barrier of j);
* consumer: wait for "ready", load block 0's out-of-block values (its
  descriptors); then for each block j: wait for it to land, write the values
  loaded for it into its buffer (its descriptors), barrier, pull, release the
  buffer, load block j+1's values (its descriptors), update block j (its
  descriptors again: the output address).

Checked on every step: descriptors are written only into ring slots no
consumer still reads; a block's copies go only into a buffer that no consumer
still writes or pulls from; a consumer writes only into a buffer no other one
still pulls an older block from, and pulls only what every consumer has
written; each read finds the descriptors of the block it wants.  The ring
sizes and buffer counts are read from the kernel headers.  The model finds
the race of a double-buffered stage with a 4-slot ring (the producer's
look-ahead then overwrites the descriptors of a block a slow consumer is still
updating), and those of a hand-over without the barrier or without "ready"."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "openludwig_b200" / "csrc"


def _const(path: Path, name: str) -> str:
    m = re.search(rf"constexpr int {name} = ([^;]+);", path.read_text())
    assert m, (path, name)
    return m.group(1).strip()


def _params():
    out = {}
    for kernel, header, ring, tab, buf in (
            ("k_sc_ws", "ws.cuh", "kWsRing", "kWsTab", "kWsBuf"),
            ("k_thermal_ws", "thermal_ws.cuh", "kTwRing", "kTwTab", "kTwBuf")):
        m = re.fullmatch(rf"(\d+) \* {buf}", _const(CSRC / header, tab))
        assert m, header  # the table follows the stage buffers
        out[kernel] = (int(m.group(1)), int(_const(CSRC / header, ring)))
    return out


class Violation(AssertionError):
    pass


def _run(buffers: int, ring: int, cnt: int, n_cons: int, rng: random.Random,
         barrier: bool = True, wait_ready: bool = True) -> None:
    slot = [None] * ring                 # block whose descriptors a slot holds
    ready = False                        # blocks 0 and 1 are described
    landed = [False] * cnt
    released = [0] * cnt                 # consumers that released block j
    written = [0] * cnt                  # consumers that wrote their values of block j
    using = [set() for _ in range(n_cons)]    # blocks whose descriptors a consumer reads
    holding = [None] * n_cons            # block whose buffer a consumer writes or pulls from

    def publish(p):
        for c in range(n_cons):
            for i in using[c]:
                if i != p and i % ring == p % ring:
                    raise Violation(f"descriptors of {p} overwrite those of {i} in use")
        slot[p % ring] = p

    def read(c, p):
        if slot[p % ring] != p:
            raise Violation(f"consumer {c} reads {slot[p % ring]} instead of {p}")

    def buffer_free_for(j, what):
        for i in holding:
            if i is not None and i != j and i % buffers == j % buffers:
                raise Violation(f"{what} {j} overwrite buffer of {i}")

    def producer():
        nonlocal ready
        publish(0)
        yield
        if cnt > 1:
            publish(1)
            yield
        ready = True
        yield
        for j in range(cnt):
            if 1 <= j and j + 1 < cnt:
                publish(j + 1)
                yield
            if j >= buffers:
                while released[j - buffers] < n_cons:
                    yield
            buffer_free_for(j, "copies of")
            landed[j] = True
            yield

    def load(c, j):                      # out-of-block values of block j into registers
        using[c].add(j)
        read(c, j)
        yield
        read(c, j)
        using[c].discard(j)

    def consumer(c):
        while wait_ready and not ready:
            yield
        yield from load(c, 0)
        for j in range(cnt):
            while not landed[j]:
                yield
            buffer_free_for(j, "values of")
            holding[c] = j
            using[c].add(j)
            read(c, j)
            yield                           # write the values
            written[j] += 1
            while barrier and written[j] < n_cons:
                yield
            if written[j] < n_cons:
                raise Violation(f"consumer {c} pulls block {j} before it is written")
            yield                           # pull
            holding[c] = None
            released[j] += 1
            yield
            if j + 1 < cnt:
                yield from load(c, j + 1)
            for _ in range(rng.randrange(1, 8)):   # the update, of varying length
                read(c, j)
                yield
            using[c].discard(j)

    actors = [producer()] + [consumer(c) for c in range(n_cons)]
    live = list(range(len(actors)))
    while live:
        a = rng.choice(live)
        try:
            next(actors[a])
        except StopIteration:
            live.remove(a)


@pytest.mark.parametrize("kernel", ["k_sc_ws", "k_thermal_ws"])
def test_protocol_never_overwrites_what_a_consumer_uses(kernel):
    buffers, ring = _params()[kernel]
    rng = random.Random(20261203)
    for _ in range(400):
        _run(buffers, ring, cnt=rng.randrange(1, 14), n_cons=3, rng=rng)


def _violated(**kw) -> bool:
    rng = random.Random(7)
    for _ in range(400):
        try:
            _run(cnt=12, n_cons=3, rng=rng, **kw)
        except Violation:
            return True
    return False


@pytest.mark.parametrize("buffers,ring", [(2, 4), (1, 3)])
def test_model_finds_the_race_of_a_short_ring(buffers, ring):
    """Too few descriptor slots for the look-ahead: two stage buffers with
    four slots, or one with three.  Some interleaving lets the producer
    overwrite a slot that a consumer still reads."""
    assert _violated(buffers=buffers, ring=ring)


@pytest.mark.parametrize("without", ["barrier", "wait_ready"])
def test_model_finds_a_missing_wait(without):
    assert _violated(buffers=2, ring=8, **{without: False})

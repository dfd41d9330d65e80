"""The ring of K and V tiles of the bias kernel as a model on the CPU.

The walk of the issuing warps is the kernel's own code (csrc/flash_attn_ring.h), compiled for the
host and recorded as a list of waits, reads and releases; the barriers, the producer and loads that
complete in any order are modelled here.  A read must find the entry that it is meant for, whatever
the order of events, and every warp must come to its end.
"""
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fast_ops_b200", "csrc")

RECORDER = r"""
#include <cstdio>
#include <cstdlib>
#include "flash_attn_ring.h"
struct Ops {
  int end;
  void wait(int slot, uint32_t parity) const { printf("w %d %u\n", slot, parity); }
  bool ready(int, uint32_t) const { return false; }
  void release(int slot) const { printf("r %d\n", slot); }
  void scores(int t, int slot) const { printf("k %d %d\n", t, slot); }
  void step(int t, int v_slot, int k_slot) const {
    printf("v %d %d\n", t, v_slot);
    if (t + 2 < end) printf("k %d %d\n", t + 2, k_slot);
  }
};
int main(int, char** a) {
  const int stages = atoi(a[1]), j0 = atoi(a[2]), j1 = atoi(a[3]), n = atoi(a[4]), first = atoi(a[5]), end = atoi(a[6]);
  if (stages == 4) fo::walk_kv_ring<4>(j0, j1, n, first, end, Ops{end});
  else fo::walk_kv_ring<6>(j0, j1, n, first, end, Ops{end});
}
"""


@pytest.fixture(scope="module")
def recorder(tmp_path_factory):
    path = tmp_path_factory.mktemp("ring")
    src, exe = str(path / "recorder.cpp"), str(path / "recorder")
    with open(src, "w") as f:
        f.write(RECORDER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, src, "-o", exe], check=True)

    def record(stages, n, halves, up):
        """The walk, up or down, of a query tile that sees `halves` half key tiles, in a ring of n key tiles."""
        own = (halves + 1) // 2
        j0 = 0 if up else n - own
        args = [stages, j0, j0 + own, n, 0 if up else halves % 2, halves if up else 2 * own]
        out = subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout
        ops = []
        for line in out.splitlines():
            kind, *num = line.split()
            num = [int(x) for x in num]
            if kind in "kv":  # a read: the entry it needs, the slot it looks in
                ops.append(("read", 2 * (j0 + num[0] // 2) + (kind == "v"), num[1]))
            else:
                ops.append(("wait" if kind == "w" else "release", *num))
        return ops

    return record


class Barrier:
    """Phases of an mbarrier: a wait for a parity returns unless the current phase has that parity."""

    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passes(self, parity):
        return self.phase & 1 != parity


def run(stages, entries, warps, rng, order):
    """Random interleaving of the producer, the warps and the loads in flight.  With `order`
    "reversed" loads complete last in, first out whenever there is a choice."""
    full = [Barrier(1) for _ in range(stages)]
    empty = [Barrier(len(warps)) for _ in range(stages)]
    held = [None] * stages  # entry in a slot; None while a load is under way
    flight, at, loaded = [], [0] * len(warps), 0

    def can_run(w):
        return at[w] < len(warps[w]) and (warps[w][at[w]][0] != "wait" or full[warps[w][at[w]][1]].passes(warps[w][at[w]][2]))

    while loaded < entries or flight or any(a < len(p) for a, p in zip(at, warps)):
        actors = [w for w in range(len(warps)) if can_run(w)]
        if loaded < entries and (loaded < stages or empty[loaded % stages].passes(((loaded // stages) & 1) ^ 1)):
            actors.append("producer")
        # loads are slow: one completes when nothing else can happen, or now and then
        if flight and (not actors or rng.random() < 0.1):
            actors = ["load"]
        assert actors, "nothing can go on"
        who = rng.choice(actors)
        if who == "producer":
            held[loaded % stages] = None
            flight.append(loaded)
            loaded += 1
        elif who == "load":
            e = flight.pop(-1 if order == "reversed" else rng.randrange(len(flight)))
            held[e % stages] = e
            full[e % stages].arrive()
        else:
            op = warps[who][at[who]]
            at[who] += 1
            if op[0] == "release":
                empty[op[1]].arrive()
            elif op[0] == "read":
                assert held[op[2]] == op[1], f"warp {who} reads entry {op[1]} in slot {op[2]}, which holds {held[op[2]]}"


@pytest.mark.parametrize("stages", [4, 6])
@pytest.mark.parametrize("order", ["random", "reversed"])
@pytest.mark.parametrize("seen0,seen1", [(1, 1), (2, 2), (2, 3), (2, 4), (3, 3), (4, 4), (4, 5), (4, 6), (5, 5), (6, 7),
                                         (6, 8), (8, 10), (11, 11), (12, 14), (17, 17), (18, 20), (19, 19)])
@pytest.mark.parametrize("up", [False, True], ids=["descending", "ascending"])
def test_every_read_finds_its_entry(recorder, stages, order, seen0, seen1, up):
    """Query tile 0 sees seen0 half key tiles, tile 1 seen1 (up to two more under a causal mask)."""
    n1 = (seen1 + 1) // 2
    warps = [recorder(stages, n1, seen, up) for seen in (seen0, seen1)]
    for warp, seen in zip(warps, (seen0, seen1)):
        assert sum(op[0] == "read" for op in warp) == 2 * seen  # K and V of every step
        assert sum(op[0] == "release" for op in warp) == 2 * n1
    for seed in range(60):
        run(stages, 2 * n1, warps, random.Random(seed), order)


def test_the_model_sees_a_wait_that_is_missing(recorder):
    """Passing over the first key tile without waiting for it lets a warp take entry 4 for loaded."""
    warps = [recorder(4, 3, seen, False) for seen in (4, 6)]
    assert warps[0][:4] == [("wait", 0, 0), ("release", 0), ("wait", 1, 0), ("release", 1)]
    del warps[0][2], warps[0][0]
    with pytest.raises(AssertionError, match="reads entry"):
        for seed in range(60):
            run(4, 6, warps, random.Random(seed), "reversed")

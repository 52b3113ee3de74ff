"""The waits of the float32 product's splitters (csrc/gemm_f32_tcgen05.cu) as a model on the CPU: two groups take slices in turn out of a
ring, barriers tell phases by their parity, copies land in any order.  Nothing may be read before it has landed, and no barrier be armed or
arrived at beyond its phase."""
import random

import pytest


class Barrier:
    def __init__(self):
        self.left, self.bytes, self.phase = 1, 0, 0

    def arrive(self, n=0):
        assert self.left > 0, "an arrival beyond the phase's"
        self.left, self.bytes = self.left - 1, self.bytes + n
        self.settle()

    def land(self, n):
        self.bytes -= n
        self.settle()

    def settle(self):
        if self.left == 0 and self.bytes == 0:
            self.left, self.phase = 1, self.phase + 1

    def done(self, parity):
        return (self.phase & 1) != parity


def walk(ring, splits, accs, waits_for_release, slices, rng):
    full, empty = [Barrier() for _ in range(ring)], [Barrier() for _ in range(ring)]
    holds, flying, split, products = [None] * ring, [], set(), set()
    copied, added, group, half = 0, 0, [0, 1], [0, 0]
    while added < slices:
        move = rng.choice(["copy", "land", "product", "add", 0, 1])
        if move == "copy" and copied < slices and (copied < ring or empty[copied % ring].done((copied // ring & 1) ^ 1)):
            full[copied % ring].arrive(1)
            flying.append(copied)
            copied += 1
        elif move == "land" and flying:
            i = flying.pop(rng.choice([0, -1]))
            holds[i % ring] = i
            full[i % ring].land(1)
        elif move == "product":
            for i in range(slices):
                if i in split and i not in products and i < added + accs and (i < 2 or i - 2 in products):
                    products.add(i)
                    break
        elif move == "add" and added in products:
            added += 1
        elif move in (0, 1) and group[move] < slices:
            it = group[move]
            s = it % ring
            if half[move] == 0:
                if waits_for_release and ring % 2 and it >= ring and not empty[s].done((it // ring & 1) ^ 1):
                    continue
                if full[s].done(it // ring & 1):
                    assert holds[s] == it, "a slice that has not landed is read"
                    half[move] = 1
            elif it < splits or it - splits in products:
                assert holds[s] == it, "a slice that has not landed is read"
                empty[s].arrive()
                split.add(it)
                group[move], half[move] = it + 2, 0


@pytest.mark.parametrize("ring, splits, accs", [(5, 4, 4), (4, 4, 4), (4, 3, 3), (3, 2, 3), (2, 2, 2)])
def test_splitters_read_what_has_landed(ring, splits, accs):
    for seed in range(300):
        walk(ring, splits, accs, True, 40, random.Random(seed))


@pytest.mark.parametrize("ring, splits, accs", [(5, 4, 4), (3, 3, 3), (3, 2, 3)])
def test_in_a_ring_of_odd_length_parity_alone_is_not_enough(ring, splits, accs):
    with pytest.raises(AssertionError):
        for seed in range(300):
            walk(ring, splits, accs, False, 40, random.Random(seed))

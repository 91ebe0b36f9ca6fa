"""Forward progress of a digit pass's look-back (sort_pass_body), simulated on
the CPU: a CTA publishes its tile's counts once it runs and waits for those of
the tiles before; CTAs start in any order, and only some are resident at a
time.  Tiles taken from a counter always finish; tiles numbered by block
index need not, so the kernel takes its tiles from the counter only."""
import os
import random
import re


def simulate(tiles, ctas, resident, seed, ticket):
    rng = random.Random(seed)
    unborn = list(range(ctas))
    rng.shuffle(unborn)
    counter, held, published, done = 0, {}, set(), 0

    def take(c):
        nonlocal counter
        if ticket:
            t, counter = counter, counter + 1
            return t
        return c
    while done < tiles:
        moved = False
        while unborn and len(held) < resident:
            c = unborn.pop()
            moved = True
            if c >= tiles:
                continue  # a surplus CTA leaves before the counter
            held[c] = take(c)
            published.add(held[c])
        for c in rng.sample(sorted(held), len(held)):
            if all(t in published for t in range(held[c])):
                moved = True
                done += 1
                if ticket and tiles > ctas and counter < tiles:
                    held[c] = take(c)
                    published.add(held[c])
                else:
                    del held[c]
        if not moved:
            return False
    return True


def test_tiles_from_a_counter_finish_in_any_start_order():
    rng = random.Random(3)
    for trial in range(300):
        ctas = rng.randint(1, 40)
        tiles = rng.randint(1, 80)
        assert simulate(tiles, ctas, rng.randint(1, ctas), trial, True), (trial, tiles, ctas)


def test_tiles_by_block_index_do_not():
    assert not all(simulate(12, 16, 4, seed, False) for seed in range(20))


def test_the_pass_takes_its_tiles_from_the_counter():
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "merge_fusion_gb300", "csrc",
                       "kifi_sort_body.cuh")
    body = open(src).read().split("sort_pass_body(", 1)[1]
    assert set(re.findall(r"\btile = ([^;]*);", body)) == {"tile_id"}
    assert set(re.findall(r"tile_id = ([^;]*);", body)) == {"sm.tile_id", "atomicAdd(&s.tile_counter[pass], 1u)"}

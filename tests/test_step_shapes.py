"""Which shapes of steps get a captured graph, played through on the host (no GPU)."""
import random

import pytest

from metallix_b200.engine.step_shapes import FAILED, StepShapes


class Played:
    """An engine's use of the policy: what happens to each step of a sequence of shapes."""

    def __init__(self, room=32, sightings=1):
        self.shapes, self.kept, self.counts = StepShapes(room, sightings), {}, {"launched": 0, "captured": 0, "replayed": 0}

    def step(self, shape):
        if not self.shapes.came(shape, self.kept):
            what = "launched"
        elif shape in self.kept:
            what = "replayed"
        else:
            what = "captured"
            if len(self.kept) >= self.shapes.room:
                least = self.shapes.least(self.kept)
                del self.kept[least]
                self.shapes.evicted(least)
            self.kept[shape] = True
        self.counts[what] += 1
        return what

    def share(self, what):
        return self.counts[what] / sum(self.counts.values())


@pytest.mark.parametrize("sightings", [1, 4])
def test_a_shape_that_comes_again_is_captured_once(sightings):
    played = Played(sightings=sightings)
    assert [played.step("a") for _ in range(7)] == ["launched"] * sightings + ["captured"] + ["replayed"] * (6 - sightings)
    assert all(played.step(n) == "launched" for n in range(100))


@pytest.mark.parametrize("shapes, replayed", [(32, 0.95), (40, 0.7), (48, 0.55), (64, 0.4)])
def test_more_recurring_shapes_than_room(shapes, replayed):
    """Captures stay rare however many shapes come again, and the steps that have a graph stay as many."""
    rng = random.Random(shapes)
    for sequence in ([rng.randrange(shapes) for _ in range(6000)], [n % shapes for n in range(6000)]):
        for sightings in (1, 4):
            played = Played(sightings=sightings)
            for shape in sequence:
                played.step(shape)
            assert played.share("captured") < 0.06 and played.share("replayed") > min(replayed, 32 / shapes - 0.1)


def test_shapes_of_another_time_make_room():
    played = Played()
    for shape in list(range(32)) * 20:
        played.step(shape)
    later = [played.step(("later", n % 8)) for n in range(1600)]
    assert "replayed" in later[-8:] and all(what == "replayed" for what in later[-8:])
    assert len(played.kept) == 32


def test_an_evicted_shape_and_one_that_failed_have_to_come_again():
    played = Played(room=1, sightings=2)
    for shape in "aaaabbbbbbbbbbbb":
        played.step(shape)
    assert set(played.kept) == {"a"} or set(played.kept) == {"b"}
    shapes = StepShapes(4, 1)
    assert [shapes.came("x", {}) for _ in range(2)] == [False, True]
    shapes.failed("x")
    assert [shapes.came("x", {}) for _ in range(FAILED + 1)] == [False] * FAILED + [True]


def test_what_is_remembered_is_bounded():
    played = Played()
    for shape in range(20000):
        played.step(shape)
    assert len(played.shapes._seen) <= 4097

"""General steps of models with state, replayed from captured graphs, against the same steps launched kernel by kernel: every
design, so every kind of state (scans, matrix memories, delta rules, the dual, lightning attention, convolutions, latent caches,
looped passes), and a capture that runs out of memory."""
import importlib

import pytest
import torch

from conftest import random_ids

pytestmark = pytest.mark.gpu
DESIGNS = ("mekazen", "zitezen", "sadosun", "dimorax", "kokolorn", "mekuvik")


def design_engine(tmp_path, design, name, dtype, **options):
    from metallix_b200.engine import Engine
    design = importlib.import_module(f"test_{design}")
    raw, seed, page, sharpen = design.MODELS[name]
    folder = str(tmp_path / name)
    if not (tmp_path / name).exists():
        (tmp_path / name).mkdir()
        design.write_folder(folder, raw, seed, sharpen)
    return Engine.from_folder(folder, dtype=dtype, page_tokens=page, num_pages=2048 // page, max_requests=8, **options), raw["vocab"]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["small", "wide"])
@pytest.mark.parametrize("design", DESIGNS)
def test_two_shapes_in_turn(tmp_path, design, name, dtype):
    """A long portion beside a decoded token, and two short ones around another, seven times each: launched, captured,
    replayed. Each advances the requests' state and pages once."""
    from metallix_b200.engine import StepEntry
    seen = {}
    for graphs in (True, False):
        engine, vocab = design_engine(tmp_path, design, name, dtype, cuda_graphs=graphs)
        long = min(70, (engine.max_context - 20) // 7)
        ids = [random_ids(300 + i, 600, vocab) for i in range(5)]
        engine.step([StepEntry("c", ids[2][:4], []), StepEntry("e", ids[4][:3], [])])
        seen[graphs] = []
        for n in range(7):
            for entries in ([StepEntry("d", ids[3][long * n:long * n + long], [0, long - 1]), StepEntry("c", [ids[2][4 + n]], [0])],
                            [StepEntry("a", ids[0][8 * n:8 * n + 8], [7]), StepEntry("e", [ids[4][3 + n]], [0]),
                             StepEntry("b", ids[1][2 * n:2 * n + 2], [0, 1])]):
                seen[graphs].append(engine.step(entries).clone())
        engine.check()
        assert not graphs or len(engine._step_graphs) == 2
    for step, (replayed, launched) in enumerate(zip(seen[True], seen[False])):
        assert torch.equal(replayed, launched), (step, float((replayed - launched).abs().max()))


@pytest.mark.parametrize("fails", ["once", "always", "otherwise"])
def test_a_capture_that_fails_leaves_the_step_to_be_launched(tmp_path, monkeypatch, fails):
    """Out of memory once: the allocator's blocks are given back and the capture is made. Always, or for another reason: the
    step runs kernel by kernel, state and pages advance once, and the next steps do not try again at once."""
    from metallix_b200.engine import StepEntry, decode_graph
    import contextlib
    capture, tries = decode_graph.capture_beside, []

    @contextlib.contextmanager
    def failing(*arguments):
        tries.append(1)
        with capture(*arguments):
            yield
            if fails == "otherwise":
                raise RuntimeError("made by the test")
            if fails == "always" or len(tries) == 1:
                raise torch.OutOfMemoryError("made by the test")

    monkeypatch.setattr(decode_graph, "capture_beside", failing)
    seen = {}
    for graphs in (True, False):
        engine, vocab = design_engine(tmp_path, "sadosun", "small", "bfloat16", cuda_graphs=graphs)
        ids = random_ids(9, 200, vocab)
        engine.step([StepEntry("c", ids[:4], [])])
        seen[graphs] = [engine.step([StepEntry("a", ids[8 * n:8 * n + 8], [7]), StepEntry("c", [ids[4 + n]], [0])]).clone()
                        for n in range(9)]
        engine.check()
        if graphs:
            assert len(engine._step_graphs) == (1 if fails == "once" else 0)
            assert len(tries) == (1 if fails == "otherwise" else 2)
        engine.manager.check_invariants()
    assert all(torch.equal(x, y) for x, y in zip(seen[True], seen[False]))


def test_a_capture_for_which_the_allocator_has_no_room(tmp_path):
    """The same with an allocator that is not given another block."""
    from metallix_b200.engine import StepEntry
    engine, vocab = design_engine(tmp_path, "sadosun", "small", "bfloat16")
    launched, _ = design_engine(tmp_path, "sadosun", "small", "bfloat16", cuda_graphs=False)
    ids = random_ids(10, 400, vocab)
    entries = [[StepEntry("a", ids[40 * n:40 * n + 40], [39])] for n in range(8)]
    want = [launched.step(step)[0].clone() for step in entries]
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        for n, step in enumerate(entries):
            if n == 4:
                torch.cuda.synchronize()
                torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
            assert torch.equal(engine.step(step)[0], want[n]), n
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    engine.check()

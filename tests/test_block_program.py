"""A block's program by itself, without a GPU: which calls it takes and what it holds.  The library's calls are stubs."""

import copy
import pickle
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from ayaka_py_b200 import ops                                     # noqa: E402
from ayaka_py_b200.cache import CacheGroupSpec                    # noqa: E402
from ayaka_py_b200.cache.manager import CacheManager              # noqa: E402
from ayaka_py_b200.cache.spec import CacheBinding                 # noqa: E402
from ayaka_py_b200.engine import program                          # noqa: E402
from ayaka_py_b200.engine.step import StepEntry, StepRunner       # noqa: E402
from ayaka_py_b200.parts.attention import Attention               # noqa: E402
from ayaka_py_b200.parts.block import PreNormBlock                # noqa: E402
from ayaka_py_b200.parts.mlp import MLP                           # noqa: E402
from ayaka_py_b200.parts.norm import LayerNorm                    # noqa: E402

WIDTH = 128


@pytest.fixture
def steps(monkeypatch):
    """The steps that the library was given."""
    given = []

    class Library:
        def ayk_program_run(self, recorded, n_ops, buffers, n_buffers, step, launched, stream):
            given.append(step._obj)
            return 0

    monkeypatch.setattr(ops, "_ready", Library)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(program, "native_allowed", lambda device: True)
    return given


def a_block():
    parts = {"norm1": LayerNorm(WIDTH, 1e-5), "mixer": Attention(WIDTH, 2, 64, 0.125), "norm2": LayerNorm(WIDTH, 1e-5),
             "ffn": MLP(WIDTH, 4 * WIDTH, "gelu_tanh")}
    for part in parts.values():
        part.bind({name: torch.zeros(d.shape) for name, d in part.tensors().items()})
    return PreNormBlock(parts)


def a_cache(block):
    return CacheManager([CacheGroupSpec("g", block.mixer.cache_need(), 1)], kv_pages=16, page_size=16, max_requests=4, max_len=64,
                        dtype=torch.float32, device="cpu")


def a_step(cache, counts=(3, 1)):
    runner = StepRunner(SimpleNamespace(device="cpu", dtype=torch.float32, max_positions=64, vocab_size=10), cache, max_tokens=64)
    slots = [cache.open(i) for i in range(len(counts))]
    cache.reserve([(s, 0, n) for s, n in zip(slots, counts)])
    return runner.prepare([StepEntry(s, 0, [0] * n) for s, n in zip(slots, counts)])


BINDING = {"mixer": CacheBinding(0, "g", 0)}


def test_a_stream_that_does_not_fit_is_refused_at_every_call(steps):
    block = a_block()
    ctx = a_step(a_cache(block))
    x = torch.zeros(4, WIDTH)
    assert block._program(x, ctx, BINDING) is None                # the first call with a cache is the parts' own
    assert block.forward(x, ctx, BINDING) is x and len(steps) == 1
    with pytest.raises(ops.KernelError, match="row width"):
        block.forward(torch.zeros(4, 100), ctx, BINDING)
    # what does not fit goes to the parts' own calls, whose checks are the same at every call
    for wrong in (torch.zeros(4, 100), torch.zeros(5, WIDTH), torch.zeros(4), torch.zeros(4, WIDTH, dtype=torch.float64),
                  torch.zeros(4, 2 * WIDTH)[:, ::2]):
        assert block._program(wrong, ctx, BINDING) is None
    ctx.req_pos0 = ctx.req_pos0.long()
    assert block._program(x, ctx, BINDING) is None and len(steps) == 1


@pytest.mark.parametrize("counts,single", [((3, 5), 0), ((1, 5, 1), 2), ((1, 1), 2)])
def test_the_partial_sums_of_single_rows_are_the_calls_own(steps, monkeypatch, counts, single):
    """Calls on two streams would meet in a buffer kept per device."""
    monkeypatch.setattr(ops, "_decode_buffer", None)
    block = a_block()
    cache = a_cache(block)
    ctx = a_step(cache, counts)
    x = torch.zeros(sum(counts), WIDTH)
    kept, empty = [], torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: kept.append(empty(*a, **k)) or kept[-1])
    assert block._program(x, ctx, BINDING) is None
    block.forward(x, ctx, BINDING), block.forward(x, ctx, BINDING)
    assert len(steps) == 2
    for step, own in zip(steps, kept[-2:]):
        assert own.data_ptr() == step.workspace and step.decode_scratch_floats == single * 2 * (64 + 2) * -(-cache.max_len // ops.DECODE_PART)
        if single:
            assert step.workspace + step.workspace_bytes <= step.decode_scratch
            assert step.decode_scratch + 4 * step.decode_scratch_floats <= step.workspace + own.numel()
    assert steps[0].workspace != steps[1].workspace


def another_forward(self, h, residual, ctx):
    return residual


CHANGES = {
    "a weight": lambda block, cache: block.ffn.bind({"up_weight": torch.ones(4 * WIDTH, WIDTH)}),
    "a weight's storage": lambda block, cache: setattr(block.norm1.weight, "data", torch.ones(WIDTH)),
    "a constant": lambda block, cache: setattr(block.norm2, "eps", 1e-6),
    "a part": lambda block, cache: setattr(block, "norm1", a_block().norm1),
    "the pages": lambda block, cache: cache.kv.__setitem__(0, tuple(t.clone() for t in cache.kv[0])),
}


@pytest.mark.parametrize("what", CHANGES)
def test_a_program_of_something_else_is_made_anew(steps, what):
    block = a_block()
    cache = a_cache(block)
    ctx = a_step(cache)
    x = torch.zeros(4, WIDTH)
    block._program(x, ctx, BINDING)
    first = block._program(x, ctx, BINDING)
    assert first is not None and block._program(x, ctx, BINDING) is first
    CHANGES[what](block, cache)
    second = block._program(x, ctx, BINDING)
    assert second is not first and block._program(x, ctx, BINDING) is second


def test_a_part_with_a_forward_of_its_own_is_not_lowered(steps):
    class Mine(MLP):
        forward = another_forward

    for change in (lambda block: setattr(block.ffn, "__class__", Mine), lambda block: setattr(block.ffn, "forward", another_forward),
                   lambda block: setattr(block, "ffn", SimpleNamespace(forward=another_forward))):
        block = a_block()
        ctx = a_step(a_cache(block))
        change(block)
        x = torch.zeros(4, WIDTH)
        assert [block._program(x, ctx, BINDING) for _ in range(3)] == [None] * 3
    # ... nor one that is given such a forward later
    block = a_block()
    ctx = a_step(a_cache(block))
    block._program(x, ctx, BINDING)
    assert block._program(x, ctx, BINDING) is not None
    block.ffn.forward = another_forward
    assert block._program(x, ctx, BINDING) is None


def test_a_block_with_programs_can_be_copied(steps):
    block = a_block()
    ctx = a_step(a_cache(block))
    x = torch.zeros(4, WIDTH)
    block._program(x, ctx, BINDING)
    assert block._program(x, ctx, BINDING) is not None
    for other in (copy.deepcopy(block), pickle.loads(pickle.dumps(block))):
        assert other.norm1 is not block.norm1 and other.norm1 is other.parts["norm1"]
        assert other._program(x, ctx, BINDING) is None            # its own first call
        assert other._program(x, ctx, BINDING) is not None


def test_a_cache_that_cannot_be_a_weak_key_leaves_the_block_to_its_parts(steps):
    block = a_block()
    ctx = a_step(a_cache(block))
    ctx.cache = SimpleNamespace(**vars(ctx.cache))
    assert [block._program(torch.zeros(4, WIDTH), ctx, BINDING) for _ in range(3)] == [None] * 3

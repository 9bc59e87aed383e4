"""A pre-norm block called by itself: the call into the library against the parts' own kernels launched one by one."""

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def a_model(dtype):
    from ayaka_py_b200.models.model import Model
    from ayaka_py_b200.registry import architecture_for
    from ayaka_py_b200.weights.loader import DictStore, load_weights
    from ayaka_py_b200 import models, parts  # noqa: F401
    gen = torch.Generator(device="cuda").manual_seed(5)
    d = 128
    config = {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "vocab_size": 64, "n_positions": 512, "n_embd": d, "n_layer": 1, "n_head": 2,
              "n_inner": 4 * d, "layer_norm_epsilon": 1e-5, "activation_function": "gelu_new"}
    arch = architecture_for(config)
    cfg = arch.config_class.from_dict(config)
    model = Model(arch.build_spec(cfg), dtype, "cuda")

    def weights():
        out = {"transformer.wte.weight": (64, d), "transformer.wpe.weight": (512, d)}
        for n in ("ln_1", "ln_2"):
            out[f"transformer.h.0.{n}.weight"] = out[f"transformer.h.0.{n}.bias"] = (d,)
        for n, r, c in (("attn.c_attn", d, 3 * d), ("attn.c_proj", d, d), ("mlp.c_fc", d, 4 * d), ("mlp.c_proj", 4 * d, d)):
            out[f"transformer.h.0.{n}.weight"], out[f"transformer.h.0.{n}.bias"] = (r, c), (c,)
        out["transformer.ln_f.weight"] = out["transformer.ln_f.bias"] = (d,)
        return {k: (torch.randn(s, generator=gen, device="cuda") * 0.1).to(dtype if len(s) == 2 else torch.float32) for k, s in out.items()}

    load = lambda: load_weights(model, DictStore(weights()), arch.normalize_name, cfg)        # noqa: E731
    load()
    return model, load


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_block_by_itself(monkeypatch, dtype):
    """Prompts, mixed steps and decode steps, the same bits; on two caches, each of which sees its weights replaced between two steps."""
    from ayaka_py_b200.cache.manager import CacheManager
    from ayaka_py_b200.engine.program import BlockProgram
    from ayaka_py_b200.engine.step import StepEntry, StepRunner
    model, load = a_model(dtype)
    block, binding = model.blocks[0], model.bindings[0]
    ran, run = [], BlockProgram.run
    monkeypatch.setattr(BlockProgram, "run", lambda self, *a: ran.append(self) or run(self, *a))
    for turn in range(2):
        cache = CacheManager(model.groups, kv_pages=64, page_size=16, max_requests=4, max_len=512, dtype=dtype, device="cuda")
        runner = StepRunner(model, cache, max_tokens=512, max_requests=4)
        slots = [cache.open(i) for i in range(3)]
        ran.clear()
        for number, counts in enumerate(([70, 33, 5], [1, 20, 1], [1, 1, 1], [40, 1, 1], [1, 1, 1])):
            if number == 3:
                load()                                   # other weights: a program that still held the old ones would show from here on
            entries = [StepEntry(s, int(cache.length[s]), [0] * n, [n - 1]) for s, n in zip(slots, counts)]
            res = cache.reserve([(e.slot, e.start, len(e.tokens)) for e in entries])
            ctx = runner.prepare(entries)
            x = torch.randn(ctx.num_rows, 128, device="cuda")
            monkeypatch.setenv("AYAKA_B200_NATIVE_STEP", "0")
            want = block.forward(x.clone(), ctx, binding)
            kept = [t.clone() for t in cache.kv[0]]
            monkeypatch.setenv("AYAKA_B200_NATIVE_STEP", "1")
            if number == 0:
                block.forward(x.clone(), ctx, binding)   # the first call with a cache is the parts' own
            assert len(ran) == number
            given = x.clone()
            got = block.forward(given, ctx, binding)
            assert len(ran) == number + 1 and got is given and torch.equal(got, want)
            assert all(torch.equal(a, b) for a, b in zip(cache.kv[0], kept))
            cache.commit(res)
        assert len(set(ran)) == 2 and ran[2] is ran[0] and ran[3] is ran[4]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_decode_steps_of_a_block_on_two_streams(dtype):
    """Their partial sums lie in memory of their own: many calls side by side give the bits of calls one after the other."""
    from ayaka_py_b200.cache.manager import CacheManager
    from ayaka_py_b200.engine.step import StepEntry, StepRunner
    model, _ = a_model(dtype)
    block, binding = model.blocks[0], model.bindings[0]
    sides = []
    for side in range(2):
        cache = CacheManager(model.groups, kv_pages=64, page_size=16, max_requests=4, max_len=512, dtype=dtype, device="cuda")
        runner = StepRunner(model, cache, max_tokens=512, max_requests=4)
        for pages in cache.kv[0]:
            pages.copy_(torch.randn(pages.shape, device="cuda"))
        slots = [cache.open(i) for i in range(3)]
        cache.commit(cache.reserve([(s, 0, 200 + 30 * i) for i, s in enumerate(slots)]))
        entries = [StepEntry(s, int(cache.length[s]), [0]) for s in slots]
        cache.reserve([(e.slot, e.start, 1) for e in entries])
        ctx = runner.prepare(entries)
        x = torch.randn(3, 128, device="cuda")
        want = [block.forward(x.clone(), ctx, binding) for _ in range(2)][1]
        sides.append((ctx, x, want, torch.cuda.Stream(), []))
    torch.cuda.synchronize()
    for _ in range(100):
        for ctx, x, _, stream, got in sides:
            with torch.cuda.stream(stream):
                got.append(block.forward(x.clone(), ctx, binding))
    torch.cuda.synchronize()
    for _, _, want, _, got in sides:
        assert all(torch.equal(y, want) for y in got)

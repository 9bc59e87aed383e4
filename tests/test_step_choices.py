"""Which kernel a step takes where more than one can: the rules that look at a step's rows and contexts, at points where both
sides were measured.  Nothing is launched."""

from types import SimpleNamespace

import numpy as np
import pytest

from ayaka_py_b200 import ops

SMS = 148


def step(plan):
    """A step's context for [(cached tokens, rows brought)], single rows first."""
    pos0, counts = (np.array(x, dtype=np.int64) for x in zip(*sorted(plan, key=lambda e: e[1] != 1)))
    return SimpleNamespace(host={"pos0": pos0, "counts": counts}, num_requests=len(plan), num_rows=int(counts.sum()),
                           num_single=int((counts == 1).sum()), max_q_len=int(counts.max()), max_kv_len=int((pos0 + counts).max()))


@pytest.mark.parametrize("heads,rank,rot,plan,tcgen05", [
    (16, 512, 64, [(0, 1024), (0, 777)], True), (16, 512, 64, [(512, 512)], True), (16, 512, 64, [(500, 2)], True),
    (16, 512, 64, [(0, 32)], False), (16, 512, 64, [(0, 64)], False), (16, 512, 64, [(20, 3)] * 200, False),
    (16, 512, 64, [(100, 1)] * 100 + [(0, 64)], False), (16, 512, 64, [(250, 3)] * 100, False),
    (16, 512, 64, [(500, 1)] * 64 + [(0, 512)], True), (8, 512, 64, [(500, 1)] * 200 + [(0, 512)], False),
    (128, 512, 64, [(0, 128)], False), (128, 512, 64, [(0, 384)], True), (130, 512, 64, [(0, 256)], False),
    (16, 256, 64, [(0, 1024)] * 2, True), (16, 256, 64, [(400, 2)] * 200, False), (40, 192, 0, [(0, 1024)] * 2, True),
    (16, 128, 64, [(0, 1024)] * 2, True), (16, 128, 64, [(0, 128)], False), (16, 64, 64, [(900, 4)] * 32, True),
    (16, 64, 0, [(0, 1024)] * 2, False)])
def test_latent_attention_takes_the_faster_of_its_tensor_core_forms(heads, rank, rot, plan, tcgen05):
    assert ops._latent_tc_pays(step(plan), heads, rank, rot, None, SMS) is tcgen05


def test_a_window_bounds_the_keys_that_a_tile_is_thought_to_read():
    ctx = step([(900, 4)] * 32)
    assert ops._latent_tc_pays(ctx, 16, 512, 64, None, SMS)
    assert not ops._latent_tc_pays(ctx, 16, 512, 64, 16, SMS)
    assert ops._latent_tiles(ctx, 8, None)[1] > ops._latent_tiles(ctx, 8, 16)[1]


@pytest.mark.parametrize("heads,dim,vdim,plan,long,apart", [
    (16, 128, 128, [(0, 64)], False, 0), (16, 128, 128, [(0, 256)], True, 0), (4, 128, 128, [(0, 64)], False, 0),
    (16, 128, 128, [(0, 1024), (0, 777)], True, 0), (16, 128, 128, [(0, 64)] * 8, True, 0), (4, 128, 128, [(0, 64)] * 8, False, 0),
    (4, 128, 128, [(0, 64)] * 64, True, 0), (16, 32, 32, [(0, 64)] * 64, False, 0), (16, 32, 32, [(0, 64)] * 250, False, 0),
    (16, 128, 128, [(9, 1)] * 8 + [(0, 64)], False, 8), (16, 128, 128, [(9, 1)] * 8 + [(0, 256)], True, 8),
    (16, 128, 128, [(9, 1)] * 250 + [(0, 64)], True, 250), (4, 128, 128, [(9, 1)] * 8 + [(0, 256)], True, 0),
    (16, 32, 32, [(9, 1)] * 64 + [(0, 64)], False, 64), (16, 128, 128, [(9, 3)] * 100 + [(0, 64)], False, 0),
    (16, 128, 128, [(9, 3)] * 30 + [(0, 256)], True, 0)])
def test_mlstm_takes_the_faster_of_its_forms_for_portions(heads, dim, vdim, plan, long, apart):
    ctx = step(plan)
    assert ops._mlstm_long_pays(ctx, heads, dim, vdim) is long
    assert ops._mlstm_singles(ctx, heads) == apart


@pytest.mark.parametrize("rows,heads,groups,tensor_cores,max_len,keys", [
    (8, 16, 4, True, 2048, 64), (8, 16, 4, True, 8192, 128), (8, 32, 8, True, 2048, 64), (32, 16, 4, True, 2048, 256),
    (32, 16, 4, True, 8192, 256), (8, 16, 16, True, 2048, 256), (128, 16, 4, True, 512, 128), (128, 16, 4, True, 100, 64),
    (32, 32, 1, True, 2048, 64), (32, 16, 4, False, 2048, 64), (128, 16, 4, False, 2048, 256)])
def test_partitions_grow_where_short_contexts_leave_no_multiprocessor_without_a_block(monkeypatch, rows, heads, groups, tensor_cores, max_len, keys):
    monkeypatch.setattr(ops, "sm_count", lambda: SMS)
    assert ops.grouped_part(max_len, ops._grouped_blocks(rows, heads, groups, 128, 128, tensor_cores)) == keys


@pytest.mark.parametrize("heads,groups,window,chunk,plan,tcgen05", [
    (16, 4, None, None, [(0, 1024)] * 2, True), (16, 4, None, 512, [(0, 1024)] * 2, True), (16, 4, None, None, [(0, 128)], True),
    (16, 4, None, None, [(0, 16)], False), (16, 4, None, None, [(500, 2)], True), (16, 4, None, None, [(500, 2)] * 32, False),
    (8, 8, None, None, [(0, 512)] * 8, True), (32, 8, None, None, [(0, 8)] * 32, False), (16, 4, None, None, [(1900, 64)], True),
    (12, 4, None, None, [(0, 128)] * 8, True)])
def test_grouped_attention_takes_the_faster_of_its_forms_for_portions(heads, groups, window, chunk, plan, tcgen05):
    assert ops._grouped_wide_pays(step(plan), heads, groups, window, chunk, SMS) is tcgen05


@pytest.mark.parametrize("heads,window,plan,expanded", [
    (16, None, [(0, 1024), (0, 777)], True), (16, None, [(0, 2)] * 2, True), (16, None, [(1900, 2)] * 2, True), (16, 512, [(1900, 300)], True),
    (16, None, [(500, 8)] * 24, False), (16, None, [(500, 2)] * 64, False), (32, None, [(500, 2)] * 24, False), (8, None, [(0, 130)] * 8, True),
    (16, None, [(500, 1)] * 64 + [(0, 512)], False), (16, None, [(40000, 512)], False), (16, None, [(500, 1)] * 4, False)])
def test_latent_attention_expands_keys_and_values_where_that_is_the_faster_form(heads, window, plan, expanded):
    """The last but one needs more scratch memory than is given; the last is a decode step."""
    pages = SimpleNamespace(shape=(4000, 16, 1, 512))
    assert ops.latent_expanded_pays(step(plan), heads, 512, window, pages, SMS) is expanded
    assert not ops.latent_expanded_pays(step(plan), heads, 512, window, SimpleNamespace(shape=(4000, 12, 1, 512)), SMS)


@pytest.mark.parametrize("requests", [1, 2, 23, 24, 25, 60])
@pytest.mark.parametrize("rows,past,most,within", [(256, 128.0, np.inf, True), (16, 8.0, 100, True), (8, 16.0, 320.0, False), (1, 0.5, np.inf, False)])
def test_sums_over_a_steps_requests_are_the_same_for_few_and_for_many(requests, rows, past, most, within):
    """Few requests are summed in a loop, many by NumPy."""
    rng = np.random.default_rng(requests)
    plan = [(int(p), int(n)) for p, n in zip(rng.integers(0, 2000, requests), rng.integers(1, 600, requests))]
    tiles = [-(-n // rows) for _, n in plan]
    keys = [min(p + n / 2 + past, most, p + n if within else np.inf) for p, n in plan]
    got = ops._portions(step(plan), rows, past, most, within)
    assert got[0] == sum(tiles) and got[1] == sum(t * k for t, k in zip(tiles, keys))
    for window in (None, 1, 70, 4096):
        held = sum(p + n - (0 if window is None else max(p - window + 1, 0) // 64 * 64) for p, n in plan)
        assert ops._latent_expanded_rows(step(plan), window) == held


def test_steps_beyond_the_grid_and_heads_that_do_not_divide_stay_with_the_other_forms():
    many = step([(0, 2)] * 65500)                          # 1,023 + 65,500 tiles of 128 rows at most
    assert not ops._grouped_wide_pays(many, 16, 4, None, None, SMS)
    assert not ops.latent_expanded_pays(step([(0, 1024)] * 65500), 16, 512, None, SimpleNamespace(shape=(4000, 16, 1, 512)), SMS)
    assert not ops._grouped_wide_pays(step([(0, 512)]), 2, 4, None, None, SMS)            # refused by the kernel's own checks
    assert not ops._grouped_wide_pays(step([(0, 512)]), 6, 4, None, None, SMS)

"""What a kernel reads of kernels in front of it, as the sources declare it.

A kernel that is launched early starts while the one in front still runs, and waits (``pdl_wait``) before it reads what
that one writes.  A load through a ``__restrict__`` parameter, or ``__ldg``, may be moved ahead of the wait by the compiler.
So those are for what no kernel of a step writes (weights, what the host uploads before the step) and, without ``const``,
for results that are only written."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "ayaka_py_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu"))

# weights and tables made from them when a model is loaded; the step's maps, uploaded by the host
WEIGHTS = {"qw", "kw", "freq", "head_bias", "mix", "gamma", "beta", "wte", "wpe", "W", "bias", "w", "norm_w", "f_bias", "lower",
           "powers", "correction", "taps_w", "w2", "b", "b2", "coeff", "mu"}
UPLOADED = {"table", "req_q_start", "req_pos0", "req_slot", "row_req", "positions", "pos", "rows"}
# results that the kernel writes and does not read
WRITTEN = {"out", "qout", "kpages", "vpages", "latent_pages", "rope_pages", "query", "ids", "weights", "sorted", "tiles",
           "row_of_pair", "w_rows1", "w_rows2", "row_scale", "partial", "raw", "nm", "scratch", "kcache", "vcache"}
READ_TOO = {("decode_mma_kernel", "kcache"), ("decode_mma_kernel", "vcache"), ("decay_chunk_scan_kernel", "scratch")}
LDG_OF = {"g4", "b4", "args.bias", "a.bias", "rows[st]"}          # the norms' and products' vectors, the experts' weight rows


def closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def kernels(text):
    """(name, parameters, body) of every kernel in a source."""
    for m in re.finditer(r"__global__", text):
        at = m.end()
        bounds = re.match(r"\s*(void\s+)?__launch_bounds__\s*", text[at:])
        if bounds:
            at = closing(text, at + bounds.end(), "()") + 1
        first = text.index("(", at)
        last = closing(text, first, "()")
        body = text.index("{", last)
        yield re.search(r"(\w+)\s*$", text[at:first]).group(1), text[first + 1:last], text[body:closing(text, body, "{}") + 1]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_only_what_no_earlier_kernel_writes_is_read_through_restrict(path):
    text = path.read_text()
    for name, parameters, body in kernels(text):
        assert "pdl_wait()" in body, f"{name} never waits for the kernel in front"
        for p in parameters.split(","):
            if "__restrict__" not in p:
                continue
            variable = re.search(r"(\w+)\s*$", p).group(1)
            if p.strip().startswith("const"):
                assert variable in WEIGHTS | UPLOADED, f"{name}: {variable} may be read ahead of the wait"
            else:
                assert variable in WRITTEN and (name, variable) not in READ_TOO, f"{name}: {variable} may be read ahead of the wait"
    for m in re.finditer(r"__ldg\((?:reinterpret_cast<[^>]*>\()?([\w.]+(?:\[\w+\])?)", text):
        assert m.group(1) in LDG_OF, f"{path.name}: __ldg of {m.group(1)}"

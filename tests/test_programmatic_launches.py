"""Kernels that are launched programmatically (pdl_wait) may be resident while the kernel ahead still
stores, so what their chain writes must not go through the non-coherent path, whose results are
defined only for memory that is read-only as long as the kernel runs.  The compiled results
cannot show the difference, so the sources are read: in these kernels and in the functions they call,
__ldg and const __restrict__ parameters name only what is constant for the whole chain, and the first
kernel behind a packing kernel is not launched programmatically."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastreg_gb300" / "csrc"

# the names that the images have in the kernels of a file and in the functions that these call
CONSTANT = {
    "fr_ref.cu": {"Tg"},
    "fr_sob.cu": {"b"},  # the cell of S in the gradient kernel
    "fr_smooth.cu": set(),
    "fr_adjoint.cu": {"S", "T"},
}
IMAGE_PARAMETER = {"load_corners": {"F"}}  # called with an image only (below)


def _functions(text):
    """(name, parameters, body) of the file's top-level functions, by braces in the first column"""
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*", "", text)
    for m in re.finditer(r"^(?!namespace|struct|constexpr|typedef|#|//)[^\n{};]*?(\w+)\(([^{};]*)\)\s*\{\n(.*?)^\}", text,
                         re.M | re.S):
        yield m.group(1), m.group(2), m.group(3)


def _ldg_bases(code):
    return set(re.findall(r"__ldg\(\s*&?(\w+(?:\.\w+)?)", code))


@pytest.mark.parametrize("name", sorted(CONSTANT))
def test_chain_fields_take_the_coherent_path(name):
    text = (CSRC / name).read_text()
    functions = {n: (params, body) for n, params, body in _functions(text)}
    chained = {n for n, (_, body) in functions.items() if "pdl_wait();" in body}
    assert chained, name
    seen, todo = set(), set(chained)
    while todo:  # the kernels and what they call
        n = todo.pop()
        seen.add(n)
        params, body = functions[n]
        allowed = CONSTANT[name] | IMAGE_PARAMETER.get(n, set())
        assert _ldg_bases(body) <= allowed, (n, _ldg_bases(body))
        restricted = set(re.findall(r"const\s+float4?\s*\*\s*__restrict__\s+(?:const\*\s*)?(\w+)", params))
        assert restricted <= allowed, (n, restricted)
        todo |= {f for f in functions if f not in seen and re.search(rf"\b{f}(<[^;()]*>)?\(", body)}


def test_load_corners_is_given_an_image():
    text = (CSRC / "fr_adjoint.cu").read_text()
    for first in re.findall(r"load_corners\((\w+),", text):
        assert first == "S", first


@pytest.mark.parametrize("fn", ["tri_checked32_3", "tri_unchecked32_f4"])
def test_shared_gathers_of_chain_fields(fn):
    body = next(b for n, _, b in _functions((CSRC / "fr_common.cuh").read_text()) if n == fn)
    assert "__ldg" not in body and "chain_load(" in body


def test_first_kernel_behind_a_packing_kernel():
    adj = (CSRC / "fr_adjoint.cu").read_text()
    assert re.search(r"launch_sob_kernel\(0, a, cuts\[0\]\.count, 0, s, k > 0\)", adj)
    api = (CSRC / "fr_api.cu").read_text()
    for fn, end in (("int autotune(fr_handle* h", "launch_iter("), ("int begin(fr_handle* h", "\n}\n")):
        body = api[api.index(fn):]
        between = body[body.index("pack_init_kernel<<<"):]
        assert "cudaMemsetAsync" in between[:between.index(end)], fn

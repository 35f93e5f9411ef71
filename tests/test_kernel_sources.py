"""Rules that hold for every kernel and whose breach shows on a GPU only now and then, if at all: read from the sources."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yalis_b200", "csrc")


def _block(text, start):
    """The text between the brace at or after ``start`` and its partner."""
    begin = text.index("{", start)
    depth = 0
    for i in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin + 1:i]
    raise ValueError("unbalanced braces")


def _kernels():
    """(name, parameters, body) of every kernel, without comments."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            head = text[m.start():text.index("{", m.start())]
            name = re.findall(r"(\w+)\s*\((?=[^()]*$|[^()]*\))", head)[-1]
            found.append((name, head[head.index(name):], _block(text, m.start())))
    return found


KERNELS = _kernels()
ids = lambda kernels: [k[0] for k in kernels]
WITH_TENSOR_MEMORY = [k for k in KERNELS if "tcgen05.alloc" in k[2]]


def test_kernels_are_found():
    assert len(KERNELS) > 50 and len(WITH_TENSOR_MEMORY) >= 4


@pytest.mark.parametrize("name,parameters,body", WITH_TENSOR_MEMORY, ids=ids(WITH_TENSOR_MEMORY))
def test_tensor_memory_is_taken_before_the_next_kernel_is_let_in(name, parameters, body):
    """One thread that lets the next kernel in does so for its block.  A block that has let it in and still waits for tensor
    memory may see a block of that kernel take the columns, which then waits for this kernel: neither ever ends."""
    alloc, let_in = body.index("tcgen05.alloc"), body.index("pdl_launch_dependents")
    assert alloc < let_in and "__syncthreads()" in body[alloc:let_in]


def _inner_loops(body):
    """The bodies of loops with braces that hold no such loop themselves."""
    for m in re.finditer(r"\bfor \(", body):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        if body[i:].lstrip().startswith("{"):
            inside = _block(body, i)
            if not re.search(r"\bfor \([^;]*;[^;]*;[^)]*\) \{[^}]*tmem_ld", inside):
                yield inside


@pytest.mark.parametrize("name,parameters,body", WITH_TENSOR_MEMORY, ids=ids(WITH_TENSOR_MEMORY))
def test_a_warp_is_whole_when_it_loads_tensor_memory(name, parameters, body):
    """The instruction asks for a converged warp: a loop whose lanes part after the load brings them together before the next."""
    for loop in _inner_loops(body):
        if "tmem_ld" in loop and re.search(r"\bif \(", loop[loop.index("tmem_ld"):]):
            assert "__syncwarp()" in loop[:loop.index("tmem_ld")], loop[:300]


# weights and other constants of a model, which no kernel of a step writes
CONSTANTS = {"w", "weight", "norm_w", "d_w", "bias", "inv_freq", "a_bias", "w_bias", "side", "table", "sink"}


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_what_another_kernel_writes_is_not_read_through_restrict(path):
    """A load through a restrict pointer may be moved above the wait for the kernel that writes what it reads."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert "__ldg" not in text
    for kind, name in re.findall(r"([\w ]+)\*\s*__restrict__\s+(\w+)", text):
        assert "const " in kind and name in CONSTANTS, (kind, name)


def test_every_bit_of_the_error_word_says_which_kernels_raise_it():
    """The bits that a source raises have a text, and a source that raises a wait's bit is of the kind that the text names."""
    import pathlib
    import re

    from yalis_b200.ops import _lib
    root = pathlib.Path(_lib.__file__).parent.parent / "csrc"
    bits = {n: int(v) for n, v in re.findall(r"YALIS_FLAG_(\w+) = (\d+)", (root / "common.cuh").read_text())}
    assert bits == {n[5:]: v for n, v in vars(_lib).items() if re.fullmatch(r"FLAG_[A-Z_]+", n)}
    kinds = {"WAIT_ATTENTION": "attention", "WAIT_PRODUCT": "gemm", "WAIT_RECURRENCE": "recurrent"}
    for source in root.glob("*.cu"):
        for name in set(re.findall(r"YALIS_FLAG_(WAIT_\w+)", source.read_text())):
            assert kinds[name] in source.name, (source.name, name)
    texts = [_lib.describe_error_word(v) for v in bits.values()]
    assert len(set(texts)) == len(bits) and not any("unknown" in t for t in texts)

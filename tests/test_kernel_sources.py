"""What the compiler has to be told about memory that another kernel writes, checked in the sources: no GPU is needed, and no run of a
kernel would show it reliably, since whether a load is moved ahead of a wait is up to the compiler.

A kernel that waits for the kernel in front (``pdl_wait``) takes that kernel's results, rows updated in place and states through pointers
without ``__restrict__``.  The names below are what may keep it.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aegean-tge_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))

# the model's constants
CONSTANTS = set("""weight weight2 q_weight k_weight kv_weight norm_weight q_norm k_norm bias cos_table sin_table conv_w conv_b a_log dt_bias
                   skip decay sink blend correction params mu mix in gain w w_up w_down""".split())
# what the host gave the step
STEP = set("positions seq_of_token q_start start_pos slots block_table pool_table rows page_seq page_idx ctx_len temperature uniform top_k top_p min_p".split())
# written, and not read before that
RESULTS = set("""out copy k_pages v_pages pages keys values latents q_latent q_out qkv act_out norm_out scaled scaled_out ss_out sums planes
                 dst gate gates qk v h inner grouped ids weights place offsets prepared""".split())
# names that mean something else elsewhere
ONLY_HERE = {("embedding_kernel", "table"), ("embedding_kernel", "ids"), ("latent_gather_kernel", "table"), ("streams_rows_kernel", "out"),
             ("streams_slices_kernel", "out")}


def functions(path: Path):
    """(name, parameters, body) of the functions defined in a source whose parameters may name pointers."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for match in re.finditer(r"__(global|device)__[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*\{", text):
        depth, at = 1, match.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        head = match.group(0)
        # the parameter list is the last one of the head (launch bounds have one of their own)
        name = re.findall(r"\b(\w+)\s*\((?!\s*\()", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", head))[0]
        yield match.group(1), name, head[head.index(name):], text[match.end():at]


def kernels(path: Path):
    return [f for f in functions(path) if f[0] == "global"]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_results_of_earlier_kernels_come_through_plain_pointers(path):
    found = []
    for kind, name, head, body in functions(path):
        if kind == "global" and "pdl_wait(" not in body:
            continue
        for const, of, pointer in re.findall(r"(const\s+)?(\w+)\s*\*\s*__restrict__\s+(\w+)", head):
            if (name, pointer) in ONLY_HERE:
                continue
            allowed = pointer in CONSTANTS or pointer in STEP if const else pointer in RESULTS
            if const and of != "int" and pointer == "rows":
                allowed = False
            if not allowed:
                found.append(f"{name}: {const}{of}* __restrict__ {pointer}")
    assert not found, found


def test_the_sources_are_read_as_they_are_meant_to_be():
    """The kernels of one file, by name: the check above must not pass because it finds none."""
    names = {name for _kind, name, _head, _body in kernels(CSRC / "gemm_tcgen05.cu")}
    assert {"gemm_tcgen05_kernel", "gemm_tcgen05_pair_kernel", "splitk_epilogue_quad_kernel", "splitk_add_norm_kernel",
            "splitk_qkv_rope_store_kernel", "splitk_add_scale_kernel"} <= names
    assert sum(len(kernels(path)) for path in SOURCES) > 90


def test_every_kernel_that_may_start_early_waits():
    """``tge_launch`` lets a kernel start while the one in front still runs: it has to wait in its own body or in a function that it calls."""
    defined, launched = {}, {}
    for path in SOURCES:
        for _kind, name, _head, body in functions(path):
            defined[name] = body
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for name in re.findall(r"tge_launch(?:_clusters)?\(\s*(?:\w+::)*(\w+)", text):
            launched.setdefault(name, path.name)
        # kernels that a launch gets through a variable or a lambda's argument
        for name in re.findall(r"(?:auto kernel =|run\(|launch\(|\?|:)\s*(\w+_kernel)\b", text):
            launched.setdefault(name, path.name)

    def waits(name):
        body = defined[name]
        return "pdl_wait(" in body or any(re.search(rf"\b{helper}(<[^;]*?>)?\(", body) and "pdl_wait(" in text for helper, text in defined.items())

    names = [name for name in launched if name in defined and name != "attention_simt_kernel"]      # that one is launched with <<< >>>
    assert len(names) > 70
    assert [name for name in names if not waits(name)] == []


def test_kernels_that_add_cuts_start_early_beside_settled_weights_only():
    """They ask for the bias ahead of their wait, which the kernel in front of the product may just have written: the product's own
    wait makes that visible to the product alone.  So without ``settled`` they are launched to start behind the whole product."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "gemm_tcgen05.cu").read_text())
    launches = re.findall(r"(\w+)\(\s*splitk_\w+_kernel\s*,\s*([^,]+),", text)
    assert len(launches) == 6 and all(how == "launch" and first.startswith("settled") for how, first in launches), launches
    assert re.search(r"void launch\([^)]*\)\([^)]*\), bool settled.*?if \(settled\) \{\s*tge_launch\(kernel", text, re.S)

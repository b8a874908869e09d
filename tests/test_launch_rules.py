"""What a kernel under programmatic dependent launch may promise about its pointers, read off the sources (no GPU).

`const T* __restrict__` tells the compiler that nothing writes the memory while the kernel runs, `__restrict__` on a pointer that is
also read that nobody else does. For what the kernel ahead in the stream writes neither holds before griddepcontrol.wait has returned:
such a load may be moved ahead of the wait or be served from a line read before it. So the qualifier may stand on weights,
tables and the step's packed input, which are in place before a step's first kernel starts, and on outputs that the kernel never
reads; every pointer that has it is named here, by file."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hipinfer_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# weights, tables, the step's packed input
CONSTANT = {
    "attention_fast.cu": "bt table row_req pos q_len ctx_len row_list r1p r2p sink",
    "attention_prefill.cu": "table",
    "attention_prefill_tc.cu": "bt q_start q_len ctx_len r1p r2p sink",
    "attention_window_flash.cu": "table",
    "core.cu": "table ptab pos w b rows scale bias slot_map bq bk bv pre_wq pre_wk temperature seed position map q_len row_req bt",
    "gemm_simt.cu": "W colscale",
    "gemm_stream_consumers.cu": "w pos slot_map table rows",
    "hyper_streams.cu": "rows a w b M a_next w_next bias",
    "latent.cu": "wq wc pos slot_map table wt row_list row_req q_len",
    "matrix_state.cu": "bi bf q_start q_len slot a_log dt_bias row_req w",
    "moe.cu": "router bias correction shared_gate w wgu wd we",
    "selective_scan.cu": "wa wb w",
    "ssd.cu": "w bias q_start q_len slot",
}
# written and never read by the kernel
OUTPUT = {
    "attention_fast.cu": "out",
    "attention_prefill_tc.cu": "out",
    "core.cu": "out y act q_out kc vc",
    "gemm_stream_consumers.cu": "y q_out kc vc",
    "hyper_streams.cu": "out xs",
    "latent.cu": "cq_out cache out dst",
    "matrix_state.cu": "a b e scal out",
    "moe.cu": "expert weight shared_weight identity_weight act out offsets pos src xs",
    "selective_scan.cu": "hi lo xb",
    "ssd.cu": "out",
}
# loads through the read-only path in so many words: of weights and block tables alone
READ_ONLY_LOADS = {
    "attention_fast.cu": ["table + pg0 + j", "row_list + tw", "table + page0 + j", "table_w + page0 + j"],
    "gemm_rows.cu": ["(const uint4*)a.norm_w + i"],
}
STREAMED = {"tc_common.cuh": "hb_ldg_stream", "moe.cu": "hb_ldg_once"}     # functions of ld.global.nc


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def closing(text, i, pair):
    """The place behind the bracket that closes the one before text[i]."""
    depth = 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
    return i


def functions(text):
    """(name, parameters, body, whether it is a kernel) of the __global__ and __device__ functions that have a body."""
    for m in re.finditer(r"__(global|device)__\s+(?:__forceinline__\s+)?[\w:<>,\s*]*?(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?"
                         r"(\w+)\s*\(", text):
        end = closing(text, m.end(), "()")
        brace = re.match(r"\s*\{", text[end:])
        if brace:
            yield m.group(2), text[m.end():end - 1], text[end:closing(text, end + brace.end(), "{}")], m.group(1) == "global"


def qualified(params):
    """(name, whether it is const) of the parameters with the qualifier."""
    return [(m.group(2), bool(m.group(1))) for m in re.finditer(r"(const\s+)?[\w:]+\s*\*\s*(?:const\s+)?__restrict__\s+(\w+)", params)]


def test_the_reader_of_the_sources_finds_the_kernels():
    found = {(f, n) for f in SOURCES for n, _, _, kernel in functions(source(f)) if kernel}
    assert len(found) == sum(len(re.findall(r"__global__", source(f))) - len(re.findall(r"__global__[^{;]*;", source(f))) for f in SOURCES)
    assert {("core.cu", "layernorm_vec_kernel"), ("moe.cu", "moe_route_kernel"), ("gemm_simt.cu", "simt_rows_kernel")} <= found
    text = "__global__ void __launch_bounds__(f(1), 2) k(const float* __restrict__ x, T *__restrict__ y, int n) { a(); }"
    assert [(n, qualified(p), k) for n, p, _, k in functions(text)] == [("k", [("x", True), ("y", False)], True)]


@pytest.mark.parametrize("name", SOURCES)
def test_no_kernel_promises_that_the_kernel_ahead_has_ended(name):
    bad = []
    for fn, params, body, kernel in functions(source(name)):
        if kernel and "hb_pdl_wait" not in body:      # starts when the kernel ahead has ended
            continue
        for p, const in qualified(params):
            if p not in (CONSTANT if const else OUTPUT).get(name, "").split():
                bad.append((fn, p))
            elif not const and any(not re.match(r"\s*=[^=]", body[closing(body, m.end(), "[]"):])
                                   for m in re.finditer(r"(?<![\w.])%s\s*\[" % p, body)):
                bad.append((fn, p, "is read"))
        bad += [(fn, m) for m in re.findall(r"__restrict__\s+\w+\s*=", body)]
    assert not bad


@pytest.mark.parametrize("name", SOURCES)
def test_read_only_loads_are_of_weights_and_tables(name):
    text = source(name)
    loads = [text[m.end():closing(text, m.end(), "()") - 1] for m in re.finditer(r"__ldg\s*\(", text)]
    assert set(loads) == set(READ_ONLY_LOADS.get(name, []))
    assert len(re.findall(r"ld\.global\.nc", text)) == (1 if name in STREAMED else 0)
    if name in STREAMED:
        assert re.search(r"%s\([^)]*\)\s*\{[^}]*ld\.global\.nc" % STREAMED[name], text)

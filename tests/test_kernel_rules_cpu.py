"""Rules of the kernels that a run on the GPU would only break now and then: read out of the sources, checked on the CPU."""
import ctypes as C
import os
import re
import subprocess

import pytest

from llmini_b200 import _ffi

CSRC = os.path.join(os.path.dirname(os.path.abspath(_ffi.__file__)), "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("last16", [False, True])
def test_one_cta_loop_stores_each_operand_buffer_once(tmp_path, last16):
    """Bulk copies of separate groups to the same memory are in no order, so the one-CTA loop may store a buffer only once, and
    has to leave in it what a launch per phase would.  Result `it` of the loop goes to buffer 1 - it % 2; the last one does so
    only where it is a 16-bit result."""
    text = _source("ns_gemm_sm100.cu")
    rule = re.search(r"constexpr bool small_keeps\(uint32_t it, uint32_t iterations, bool last16\) \{[^}]*\}", text)
    assert rule and "store_panels((it & 1u) ? x0_map : x1_map" in text
    assert re.search(r"if \(issuer && !fp32 && small_keeps\(it, loop\.iterations, loop\.last16 != 0\) && elect_one\(\)\)\s*store_panels", text)
    src, lib = tmp_path / "rule.cpp", tmp_path / "rule.so"
    src.write_text("#include <cstdint>\n" + rule.group(0) +
                   '\nextern "C" int keeps(uint32_t it, uint32_t n, int l) { return small_keeps(it, n, l != 0); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    keeps = C.CDLL(str(lib)).keeps
    for iterations in range(1, 9):
        results = [it for it in range(iterations) if last16 or it + 1 < iterations]   # in 16 bits
        per_phase = {}
        for it in results:
            per_phase[1 - it % 2] = it
        stored = [it for it in results if keeps(it, iterations, int(last16))]
        assert len({1 - it % 2 for it in stored}) == len(stored), (iterations, stored)
        assert {1 - it % 2: it for it in stored} == per_phase, (iterations, stored)


def _function(text, name):
    """The body of a function of the source, without its closing brace."""
    head = re.search(r"\b" + name + r"\([^;{]*\{", text)
    assert head, name
    depth, at = 1, head.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return text[head.end():at - 1]


def test_transform_scalars_are_read_past_l1():
    """The launches of the one-tensor chain resolve the transform's scalars before they wait for the launch in front of them:
    L1 may still hold what an earlier kernel of the stream saw of these trained values."""
    body = _function(_source("stream_kernels.cu"), "symexp_resolve")
    reads = re.findall(r"(\S*)\(?p\.scales\[2 \* k[^\]]*\]\)?", body)
    assert reads and all(r.startswith("__ldcg(") for r in reads), reads


def test_column_statistics_read_past_l1():
    """k_normuon_stats_columns reads before it waits: its tables, the Newton-Schulz result, the weights and the old second
    moments all come from L2."""
    text = _source("stream_kernels.cu")
    body = _function(text, "normuon_stats")
    head, rest = body.split("if (!COLS) {", 1)
    columns = rest[rest.index("const uint32_t quad = tid % kQuads"):]
    for table in (r"slots\[", r"nv\.unit_prefix\b", r"\bu_ptrs\b", r"nv\.factor_ptrs\b"):
        reads = re.findall(r"(\S*?)&?" + table, head)
        assert reads and all(r.endswith("normuon_load<COLS>(") for r in reads), (table, reads)
    assert "slots[" not in columns and "*reinterpret_cast<const" not in columns
    assert re.findall(r"\bstate\[col\]\s*(\S+)", columns) == ["="]
    assert "0.95f * __ldcg(state + col)" in columns
    assert re.findall(r"(\w+\()?\b[Uz] \+", columns) == ["ld_l2(", "ld_l2("]
    assert '"ld.relaxed.gpu.global.v4.f32' in _function(_source("common.cuh"), "ld_l2")
    assert "return COLS ? __ldcg(p) : *p;" in _function(text, "normuon_load")


def _kernel(text, name):
    """(parameters, body) of a kernel."""
    head = re.search(r"__global__[^;{]*\b" + name + r"\(([^{]*)\)\s*\{", text)
    assert head, name
    return head.group(1), _function(text, name)


def _check_early_reader(text, name):
    """A kernel that lets the next launch begin and reads before it waits: it waits in every block, in front of that it stores
    nothing to global memory, and reads it from L2 only."""
    params, body = _kernel(text, name)
    assert body.count("chain_wait();") == 1, name
    early, late = body.split("chain_wait();")
    assert "return" not in early, name
    depth = early.count("{") - early.count("}")      # the wait itself: by every thread, or by the first of every block
    assert depth == 0 or (depth == 1 and re.search(r"if \(tid == 0\) \{[^{}]*(\{[^{}]*\}[^{}]*)*$", early)), name
    early = re.sub(r"\bsymexp_resolve\(sp, beta\)|encode_fetch<MODE, true>\(r, src, z, xm, len, base\)", "", early)
    for param in params.split(","):
        if "*" not in param:
            continue
        pointer = param.split("*")[-1].strip()
        uses = re.findall(r"(.{0,48})(?<![\w.])" + pointer + r"\b", early)
        assert all(re.search(r"__ldcg\(reinterpret_cast<const \w+ \*>\($", u) for u in uses), (name, pointer, uses)


def test_launches_that_read_before_they_wait():
    """What is launched by launch_chained may begin while the launch in front runs (csrc/stream_kernels.cu).  The first of a chain
    waits and only then lets the next one begin, so that a launch that has begun finds every input of the call written; the
    others are early readers.  The column statistics are the exception: they store before they wait, to slots that no launch in
    flight looks at (the row statistics in front of them work on the other slots), and the plain launch of these is what their
    inputs are complete before; all that they read is checked in test_column_statistics_read_past_l1."""
    text = _source("stream_kernels.cu")
    launched = re.findall(r"launch_chained\((k_\w+)", text)
    assert sorted(set(launched)) == ["k_chain_chunk_amax", "k_chain_encode", "k_chain_schedule_amax", "k_chain_zero", "k_normuon_stats_columns"]
    first = {name: re.match(r"\s*(\w+\(\);)", _kernel(text, name)[1]).group(1) for name in launched}
    heads = {name for name in launched if first[name] == "chain_head();"}
    assert heads == {"k_chain_zero", "k_chain_chunk_amax"}
    assert re.fullmatch(r"\s*chain_wait\(\);\s*chain_begin\(\);\s*", _function(text + _source("common.cuh"), "chain_head"))
    for name in set(launched) - heads:
        assert first[name] == "chain_begin();", name
        if name != "k_normuon_stats_columns":
            _check_early_reader(text, name)
    # a chain begins with its head ...
    chain = _function(text, "launch_quantize_chain")
    for branch in (chain[chain.index("if (src) {"):chain.index("return e;")], chain[chain.index("return e;"):]):
        assert re.search(r"launch_chained\((k_\w+)", branch).group(1) in heads
    # ... and the column statistics follow those of the rows, a plain launch of a kernel that waits in its first statement
    assert re.search(r"stream_launch\(kPlain, k_normuon_stats_rows,[^;]*;\s*if \(nv\.columns\) launch_chained\(k_normuon_stats_columns,",
                     _function(text, "launch_normuon_stats"))
    assert re.fullmatch(r"\s*chain_begin\(\);\s*normuon_stats<1>\([^;]*\);\s*chain_wait\(\);\s*", _kernel(text, "k_normuon_stats_columns")[1])
    assert re.fullmatch(r"\s*stream_enter\(\);\s*normuon_stats<0>\([^;]*\);\s*", _kernel(text, "k_normuon_stats_rows")[1])
    # what the early readers share
    fetch = _function(text, "encode_fetch")
    direct, bounded = fetch.split("return;", 1)
    assert re.search(r"if \(!L2_ONLY && ", direct)
    assert re.findall(r"(L2_ONLY \? __ldcg)?\(?[^?;]*: ld_stream\((\w+) \+ e\)", bounded) == [("L2_ONLY ? __ldcg", p) for p in ("src", "z", "xm")]
    assert "ld_stream" not in re.sub(r"L2_ONLY \? __ldcg\(reinterpret_cast<const float4 \*>\(\w+ \+ e\)\) : ld_stream\(\w+ \+ e\)", "", bounded)

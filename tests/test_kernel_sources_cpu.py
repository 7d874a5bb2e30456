"""Rules of the overlapped launches that a run cannot show, read off the sources."""

import glob
import importlib.util
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "flash-topk-attention_b200", "csrc")


def _functions():
    """name -> (source of the declaration and body, is it a kernel), comments taken out."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"^(?:template <[^;{}]*>\s)?[^\n;{}#]*\b(__global__|__device__)\b[^;{}]*\{",
                             text, re.M):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            head = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)|__cluster_dims__\([^()]*\)", "",
                          m.group(0))
            name = re.search(r"(\w+)\s*\(", head)
            if name:
                out.setdefault(name.group(1), (text[m.start():end], m.group(1) == "__global__"))
    return out


FUNCTIONS = _functions()
KERNELS = {n: s for n, (s, kernel) in FUNCTIONS.items() if kernel}
OVERLAPPED = sorted(n for n, s in KERNELS.items() if "pdl_wait()" in s or "dkv_union(" in s)


def test_the_sources_are_understood():
    assert {"score_kernel", "sparse_fwd_kernel", "sparse_fwd_pipe_kernel", "sparse_fwd_pipe2_kernel",
            "sparse_bwd_dq_kernel", "sparse_bwd_dq2_kernel", "sparse_bwd_dq256_kernel",
            "sparse_bwd_dkv_kernel", "sparse_bwd_dkv2_kernel", "sparse_bwd_dkv256_kernel",
            "topk_select_reg_kernel", "qblock_merge_warp_kernel", "fan_in_kernel", "head_sum_kernel",
            "cast_bf16_kernel"} <= set(OVERLAPPED)


@pytest.mark.parametrize("name", [n for n in OVERLAPPED if "tmem_alloc" in KERNELS[n]])
def test_tmem_is_allocated_before_the_next_kernel_may_start(name):
    """tcgen05.alloc waits without a limit: between it and the trigger of the successor,
    whose blocks may take the columns and keep them until this grid is done, there is a
    barrier of the block."""
    barrier = r"__syncthreads\(\)|build_union(?:_masks)?\b[^;]*;"
    for helper in ("build_union", "build_union_masks"):
        assert "__syncthreads()" in FUNCTIONS[helper][0]
    body = KERNELS[name]
    assert "pdl_launch()" in body or "dkv_union(" in body
    if "dkv_union(" in body:
        union = FUNCTIONS["dkv_union"][0]
        assert re.search(barrier, union[:union.index("pdl_launch()")])
        assert "tmem_alloc" in body[:body.index("dkv_union(")]
    if "pdl_launch()" in body:
        first = body.index("pdl_launch()")
        alloc = body.index("tmem_alloc")
        assert alloc < first, "the successor may start before the columns are taken"
        assert re.search(barrier, body[alloc:first]), "no barrier between allocation and trigger"


@pytest.mark.parametrize("name", OVERLAPPED)
def test_kernels_wait_before_their_successor_may_start(name):
    """A successor may rely on its predecessor's predecessor: where a kernel waits for the one
    before it first and only then allows the next one, that is over."""
    body = KERNELS[name]
    trigger = re.search(r"pdl_launch\(\)|dkv_union\(", body)
    assert trigger and "pdl_wait()" in body[:trigger.start()]
    if name != "score_kernel":
        assert not re.search(r"if \(!?p\.\w+\) pdl_wait", body), "a wait that a launch may leave out"


def test_the_launch_that_waits_at_its_end():
    """The second scoring launch of a call touches memory before it waits.  Its predecessor has
    to be the first one, which waits ahead of its trigger, and each of its own blocks has to wait
    all the same, as the last thing that it does."""
    body = KERNELS["score_kernel"]
    assert re.findall(r"[^\n;{}]*pdl_wait\(\)", body) == ["  if (!p.behind) pdl_wait()",
                                                        "  if (p.behind) pdl_wait()"]
    assert re.search(r"if \(!p\.behind\) pdl_wait\(\);\s*pdl_launch\(\);", body)
    assert re.search(r"if \(p\.behind\) pdl_wait\(\);\s*\}\s*$", body)
    assert not re.search(r"\breturn;", body), "a block that leaves early breaks the chain"
    text = "".join(re.sub(r"//[^\n]*", "", open(f).read()) for f in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(re.findall(r"\bbehind\b", text)) == 4   # the field, the two waits, one launch
    host = re.search(r"launch_pdl\(score_kernel<D, false>[^;]*;(.*?)p\.behind = 1;\s*return clusters\(", text,
                     re.S)
    assert host and re.sub(r"\s+", " ", host.group(1)).strip() == (
        "if (split.tail == 0) return FTK_OK; p.tile0 = static_cast<int>(first);")


def test_no_read_only_loads_in_overlapped_kernels():
    """ld.global.nc (__ldg, const __restrict__ parameters) is defined only for memory that
    does not change during the kernel's life; an overlapped kernel's inputs are written by
    the kernel it overlaps.  Kernels that are launched behind the whole of their
    predecessor may use them; whatever else is in the sources, helpers included, may not."""
    text = ""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text += re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
    for n in KERNELS:
        if n not in OVERLAPPED:
            assert KERNELS[n] in text
            text = text.replace(KERNELS[n], "")
    for what in (r"__ldg\b", r"\b__restrict__\b", r"ld\.global\.nc"):
        assert not re.search(what, text), what
    launched = set(re.findall(r"(\w+)(?:<[^<>;]*>)?<<<", text))
    assert not launched & set(OVERLAPPED), "an overlapped kernel must be launched as one"


@pytest.mark.parametrize("helper", ["cluster_arrive", "cluster_wait"])
def test_aligned_cluster_barriers_converge_first(helper):
    """barrier.cluster.*.aligned is undefined unless all threads of a warp execute it together;
    the kernels get there behind branches of single threads and loops whose trip count differs
    between the lanes.  Nothing but the helpers, which converge the warp, names it."""
    body = FUNCTIONS[helper][0]
    assert re.search(r"__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.\w+\.\w+\.aligned", body)
    text = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(re.findall(r"barrier\.cluster\.", text)) == 2


def test_registers_suffice():
    """Kernels whose loop over the tiles has 96 registers a thread put at most 96 bytes of
    them into local memory (what ptxas reports at the build; a few words around the prologue
    do no harm).  The exact forward, a fallback, may hold two accumulators' worth more."""
    spec = importlib.util.spec_from_file_location("ftk_build", os.path.join(os.path.dirname(CSRC), "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    seen = 0
    for src in ("score.cu", "sparse_fwd.cu", "sparse_bwd.cu"):
        if not os.path.exists(build.ptxas_log(src)):
            pytest.skip("not built here")
        text = open(build.ptxas_log(src)).read()
        for name, spilled in re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores", text,
                                        re.S):
            seen += 1
            assert int(spilled) <= (192 if "17sparse_fwd_kernel" in name else 96), name
    assert seen > 40

"""Orders that a wait in a kernel depends on and that no output shows: read from the kernels' sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "nano-vllm-moe_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh")}


def body(source, function):
    """The text between the braces of one function of a source."""
    at = source.index("{", source.index(f" {function}("))
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return source[at:i]
    raise AssertionError(f"{function} does not end")


def test_pair_tensor_memory_is_taken_and_released_while_both_ctas_are_there():
    """tcgen05.alloc / dealloc of a CTA pair are collective over both CTAs: the partner has to run, and has to be there still."""
    common = SOURCES["umma_common.cuh"]
    begin, release, leave = (body(common, f) for f in ("pair_tmem_begin", "pair_tmem_release", "pair_leave"))
    assert "cluster_sync_all" in body(common, "pair_enter")
    assert begin.index("tmem_alloc_pair") < begin.index("__syncthreads")
    assert release.index("mbar_wait<true>") < release.index("__syncwarp") < release.index("tmem_dealloc_pair")
    assert leave.index("__syncthreads") < leave.index("cluster_sync_all")
    rows = {"umma_pair_gemm.cu": "&tmap_a, kb", "umma_w8a8_pair.cu": "load_rows(it0", "umma_w8a16_pair.cu": "&tmap_x, kb"}
    for name, text in SOURCES.items():
        rest = text.replace(begin, "").replace(release, "")
        assert not re.findall(r"(?<!void )tmem_(?:de)?alloc_pair\(", rest), f"{name} takes or releases a pair's tensor memory by itself"
        assert ("= pair_tmem_begin(" in text) == (name in rows)
    for name, load in rows.items():
        text = SOURCES[name]
        order = ["mbar_init(", "pair_enter();", "= pair_tmem_begin(", "pair_tmem_release(", "pair_leave();"]
        at = [text.index(o) for o in order]
        assert at == sorted(at) and all(text.count(o) == 1 for o in order if o not in ("mbar_init(", "pair_tmem_release(")), (name, at)
        # once per launch: split-K releases under its band of sums, the others in the issuer's role
        assert text.count("if (!kSplit) pair_tmem_release(") == text.count("pair_tmem_release(") - 1, name
        # the partner's rows, which a leader's MMA waits for, are loaded behind the partner's own allocation
        assert at[2] < text.index(load), name
        # every role that uses tensor memory says when it is done, once per warp: epilogue, and converters where there are any
        users = 2 if "kConvWarps" in text else 1
        assert text.count("pair_tmem_done(") == users, name
        assert ("2 * (kConvWarps + kEpiWarps)" if users == 2 else "2 * kEpiWarps") + ");\n        s_abort" in text, name


def test_named_barriers_do_not_ask_for_a_converged_warp():
    """The aligned form (bar.sync, or barrier.cta with .aligned) needs the whole warp at the instruction; the epilogues come there
    out of branches that one lane took."""
    for name, text in SOURCES.items():
        asm = re.findall(r'"[^"\n]*\b(?:bar\.(?:sync|red|arrive)|barrier\.cta\.[a-z.]+)[^"\n]*"', text)
        if name == "umma_common.cuh":
            assert len(asm) == 2 and not any("bar.sync" in a or ".aligned" in a for a in asm), asm
        else:
            assert not asm, f"{name}: {asm}"


def waiting_kernels():
    """(file, name, signature, body) of every kernel that waits for the one in front of it."""
    for name, text in SOURCES.items():
        for head in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\(", text):
            rest = " " + text[head.end(1) - len(head.group(1)):]
            code = body(rest, head.group(1))
            if "pdl_wait(" in code:
                yield name, head.group(1), rest[:rest.index("{")], code


def test_only_packed_weights_are_read_before_the_wait_for_the_kernel_in_front():
    """A bias or a norm's weight may be a copy that the caller's last kernel wrote; only griddepcontrol.wait orders it."""
    early = re.compile(r"\b(bias|weight|w_scale|input_scale|h_scale|topk_w|residual)\b")
    found = {}
    for file, kernel, _, code in waiting_kernels():
        before = re.sub(r"if \([^;{]*\) prefetch_l2\([^;]*;|prefetch_l2\([^;]*;", "", code[:code.index("pdl_wait(")])
        found[file, kernel] = early.findall(before)
    assert len(found) > 15 and not any(found.values()), {k: v for k, v in found.items() if v}


def test_nothing_but_weights_goes_through_the_read_only_path():
    """Read-only loads promise that nobody writes the memory while the kernel runs, and the assembler moves them in front of the
    wait for the kernel that does: packed weights alone may take that path."""
    weights = {"stream_kernel.cu": ["wa + tile_off(k)", "wb + tile_off(k)"], "elementwise.cu": ["src + off"]}
    for name, text in SOURCES.items():
        if name == "common.cuh":
            assert len(re.findall(r"ld\.global\.nc", text)) == 1 and "ld.global.nc" in body(text, "ld_stream16")
            text = text.replace(body(text, "ld_stream16"), "")
            assert "ld.global.nc" not in text
        else:
            assert re.findall(r"ld_stream16\(([^;]*)\);", text) == weights.get(name, []), name
            assert "ld.global" not in text, name
        assert not re.search(r"__ld(?:g|cg|ca|cs|lu|cv)\(", text), name
    for file, kernel, signature, code in waiting_kernels():
        for pointer in re.findall(r"const (?:\w+|\w+ \w+)\* __restrict__ (\w+)", signature):
            assert not re.search(rf"\b{pointer}\[|\*{pointer}\b", code), f"{file}: {kernel} reads {pointer} plainly"


def test_tensor_memory_is_handed_over_at_cluster_scope():
    """A barrier that another CTA arrives on is named at cluster scope on both sides: the arrival and the wait."""
    common = SOURCES["umma_common.cuh"]
    assert "mbarrier.arrive.relaxed.cluster.shared::cluster" in body(common, "mbar_arrive_remote")
    assert "mbarrier.try_wait.parity.relaxed.cluster.shared::cta" in body(common, "mbar_wait")
    for name in ("umma_pair_gemm.cu", "umma_w8a8_pair.cu", "umma_w8a16_pair.cu"):
        remote = set(re.findall(r"(bar_\w+)\[", " ".join(re.findall(r"mbar_arrive_remote\([^;]*;", SOURCES[name]))))
        remote |= {"bar_conv"} if "conv0" in SOURCES[name] else set()
        assert "bar_tempty" in remote, name
        for bar in remote:
            waits = re.findall(r"(mbar_wait(?:<true>)?)\(smem_u32\(&" + bar, SOURCES[name])
            assert waits and set(waits) == {"mbar_wait<true>"}, (name, bar, waits)


def test_cluster_barriers_are_reached_by_warps_that_are_together():
    """The two instructions stand in one place each, behind a __syncwarp: a loop that part of a warp skips may end at the call."""
    for name, text in SOURCES.items():
        found = re.findall(r"barrier\.cluster\.\w+[.\w]*", text)
        if name != "umma_common.cuh":
            assert not found, (name, found)
    for function, instruction in (("cluster_arrive", "barrier.cluster.arrive.release.aligned"), ("cluster_wait", "barrier.cluster.wait.acquire.aligned")):
        code = body(SOURCES["umma_common.cuh"], function)
        assert code.index("__syncwarp()") < code.index(instruction)
    assert len(re.findall(r"barrier\.cluster\.", SOURCES["umma_common.cuh"])) == 2


def test_grouped_pairs_take_and_release_tensor_memory_as_the_other_pair_kernels_do():
    text = SOURCES["umma_grouped_pair.cu"]
    order = ["mbar_init(", "pair_enter();", "pair_tmem_begin(", "pdl_wait();", "&maps.w, 0, wr.a", "pair_tmem_release(", "pair_tmem_done(", "pair_leave();"]
    at = [text.index(o) for o in order]
    assert at == sorted(at) and all(text.count(o) == 1 for o in order if o != "mbar_init("), at
    assert "2 * kEpiWarps);\n        s_abort" in text
    # every item's tensor memory is handed on at cluster scope: arrivals of both CTAs, one wait
    assert re.findall(r"(mbar_wait(?:<true>)?)\(smem_u32\(&bar_tfree", text) == ["mbar_wait<true>"]
    assert text.count("mbar_arrive_remote(free_bar)") == 2 and "map_to_cta(smem_u32(&bar_tfree[side]), 0)" in text

"""Rules of the kernels that keep a failed launch from spreading, read off the CUDA sources: what they guard against cannot be
made to happen on a GPU that others share."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vtpack_b200", "csrc")
WAITING = {"linear_tc_kernel": "linear_tc.cu", "linear_tc_small_kernel": "linear_tc.cu", "attn_tc_kernel": "attention_tc.cu",
           "linear_f32_tc_kernel": "linear_f32_tc.cu", "linear_f32_terms_kernel": "linear_f32_terms.cu",
           "attn_f32_tc_kernel": "attention_f32_tc.cu", "mlp_tc_kernel": "mlp_tc.cu",
           "linear_tc_pair_kernel": "linear_tc.cu"}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"/\*.*?\*/", " ", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def body(name, text):
    """From the opening brace of function `name` to the one that closes it."""
    at = text.index("{", re.search(r"\b%s\(" % name, text).start())
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i]
    raise AssertionError(name)


@pytest.mark.parametrize("kernel", sorted(WAITING))
def test_stores_hang_on_a_status_word_read_behind_the_wait(kernel):
    """Nothing is written after a launch that gave up on a wait.  The kernel in front, which may be the one that gives up, has
    completed only behind griddepcontrol.wait, so the last look at the word lies there; and two threads that look for themselves
    can decide differently, so every look is one thread's."""
    text = body(kernel, source(WAITING[kernel]))
    looks = [m.start() for m in re.finditer(r"launch_is_void\(", text)]
    assert len([at for at in looks if at > text.index("pdl_begin()")]) == 1
    for at in looks:
        guard = max(m.end() for m in re.finditer(r"if \(threadIdx\.x == ([^()]|\([^()]*\))*\)", text[:at]))
        assert ";" not in text[guard:at] and "{" not in text[guard:at]


def test_no_other_code_looks_at_the_wait_codes():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".h", ".cuh")) and name != "common.cuh":
            assert "STATUS_WAIT_MASK" not in source(name), name


def test_device_arrays_state_their_alignment():
    """An array of the library's own is aligned to its element type unless it says more, and the kernels read such arrays through
    vector types (the linker happens to align them well enough: nothing else would show it)."""
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".h", ".cuh")):
            for line in re.findall(r"^(?:static )?__device__ (?!__forceinline__)[^;{]*\[[^;]*;", source(name), flags=re.M):
                said = re.search(r"(?:__align__|alignas)\((\d+)\)", line)
                assert said and int(said.group(1)) >= 16, (name, line)
                found += 1
    assert found >= 2


@pytest.mark.parametrize("stages", range(3, 9))
def test_pair_producers_wait_for_every_last_commit(stages):
    """Before a CTA of a pair ends, its producers wait for the commit of every stage's last fill.  A wait goes by the parity of a
    barrier's phase, so it means what it says only if the commit before has been seen: here the MMA thread is as late as the
    waits in front allow, and no wait may pass on an older commit."""
    text = body("linear_tc_kernel", source("linear_tc.cu"))
    drain = text[text.index("if (CG == 2 && ok"):text.index("rank == 0 && elect_one()")]
    own = re.search(r"f % PRODUCERS == \(uint32_t\)warp", drain) is not None      # else producer 0 waits for all, by stage
    producers = 3
    for filled in range(1, 6 * stages):
        last = sorted(range(max(0, filled - stages), filled), key=lambda f: f if own else f % stages)
        waited = set()
        for w in range(producers):
            mine = [f for f in range(filled) if f % producers == w]
            done = mine[-1] - stages + 1 if mine else 0         # k-blocks committed for sure: all up to the last one waited for
            for f in last:
                if own and f % producers != w or not own and w != 0:
                    continue
                phases = len(range(f % stages, max(done, 0), stages))
                passes = (phases - 1) & 1 == (f // stages) & 1     # (a fresh barrier passes a wait on parity 1)
                assert not passes, (filled, w, f)
                done = f + 1                                     # commits are in order
                waited.add(f)
        assert waited == set(last)


def elected_spans(text):
    """What one elected thread runs of a kernel."""
    spans = []
    for m in re.finditer(r"if \((rank == 0 && )?elect_one\(\)\) \{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        spans.append((m.end(), i))
    return spans


def test_the_rings_of_the_mlp_are_one_thread_s():
    """The waits of the rings of W stand in their methods: each is a thread's own, and every call of those methods is one elected thread's."""
    text = source("mlp_tc.cu")
    methods = body("WRing", text[:text.index("struct MlpConf")].replace("struct WRing {", "struct WRing( {"))
    waits = re.findall(r"\bmbar_(\w*wait\w*)\(", methods)
    assert len(waits) >= 4 and set(waits) == {"wait_a", "try_wait_a"}
    kernel = body("mlp_tc_kernel", text)
    spans = elected_spans(kernel)
    calls = [m.start() for m in re.finditer(r"\bw[12]?\.(load|drain|ready|mma|done)\(", kernel)]
    assert len(calls) >= 10 and all(any(a <= at < b for a, b in spans) for at in calls)


@pytest.mark.parametrize("stages", range(1, 9))
def test_ring_loader_waits_for_every_last_commit(stages):
    """The same for the rings of the one-launch MLP: one loader, which has seen the commits of all but the last fill of every stage."""
    drain = body("drain", source("mlp_tc.cu"))
    assert "d = n > (uint32_t)STAGES ? n - STAGES : 0; d < n; ++d" in drain
    wait = re.search(r"mbar_wait_a\(empty \+ 8 \* \((.*?)\), (.*?), c\.abort_flag", drain)
    stage, parity = (e.replace("/", "//") for e in wait.groups())
    for n in range(1, 6 * stages):
        seen = max(0, n - stages)                              # commits of the fills in front of these
        for d in range(max(0, n - stages), n):
            names = dict(d=d, STAGES=stages)
            assert eval(stage, {}, names) == d % stages
            phases = len(range(d % stages, seen, stages))
            assert (phases - 1) & 1 != eval(parity, {}, names)          # passes on no older commit
            assert phases & 1 == eval(parity, {}, names)                # and on this fill's
            seen = d + 1


@pytest.mark.parametrize("stages", [6, 8])
def test_shared_tile_commits_only_what_a_producer_waits_for(stages):
    """linear_tc_pair_kernel has no drain: a stage is committed only where a later fill waits for it, in both CTAs."""
    text = body("linear_tc_pair_kernel", source("linear_tc.cu"))
    commits = re.findall(r"if \((.*?)\) umma_commit_a<2>\(empty_a", text)
    waits = re.findall(r"if \((.*?) && !mbar_wait_a\(empty_a \+ 8 \* s, \(\(i / STAGES\) & 1\) \^ 1", text)
    assert commits == ["i + STAGES < n_stages"] and waits == ["i >= STAGES"]
    for n in range(1, 6 * stages):
        committed = {i for i in range(n) if i + stages < n}
        assert committed == {i - stages for i in range(n) if i >= stages}


@pytest.mark.parametrize("kernel", sorted(WAITING))
def test_lanes_that_wait_together_go_on_together(kernel):
    """A wait gives up after about a second, lane by lane.  Where a whole warp waits, warp-wide instructions follow, which a lane
    that went to unwind never reaches: such waits are decided by a vote, or no lane leaves.  Others are those of one elected thread."""
    text = body(kernel, source(WAITING[kernel]))
    elected = elected_spans(text)
    waits = [(m.start(), m.group(1)) for m in re.finditer(r"\bmbar_(\w*wait\w*)\(", text)]
    assert len(waits) >= 3
    for at, name in waits:
        one = any(a <= at < b for a, b in elected)
        # (the warps that split fp32 operands have only __syncwarp behind it, which a lane that leaves still runs as often)
        runs_out = "num_kb - kb; n > 0; --n) __syncwarp();" in text[at:at + 400]
        assert name in (("wait", "wait_a", "try_wait_a") if one or runs_out else ("wait_warp", "wait_cluster_warp")), (name, text[at:at + 80])


def test_no_mma_is_issued_in_front_of_the_fence_behind_a_wait():
    """What a wait on an mbarrier says about tensor memory (an accumulator was read, an operand is there) holds for an MMA only behind
    tcgen05.fence::after_thread_sync.  The one-launch MLP has it in ``ready``, which stands in front of every MMA: on every way through
    that goes on, and with no further wait between.  (No MMA and no wait can be made late enough on purpose to show the order.)"""
    text = source("mlp_tc.cu")
    ready = body("ready", text)
    ways = [m.start() for m in re.finditer(r"return true;", ready)]
    assert ways and all("tc_fence_after_sync()" in ready[:at] for at in ways)
    kernel = body("mlp_tc_kernel", text)
    mmas = [m.start() for m in re.finditer(r"\bw[12]\.mma\(", kernel)]
    assert len(mmas) >= 4
    for at in mmas:
        assert kernel.rfind(".ready(", 0, at) > max(kernel.rfind("mbar_wait", 0, at), kernel.rfind(".done(", 0, at))


def test_shared_memory_is_reserved_for_the_largest_launch():
    """A kernel's limit of shared memory is set once per device.  Set to what a launch takes that depends on the call, a thread could
    lower what another has just raised for a larger batch and is about to launch with."""
    for name in ("attention_tc.cu", "attention_f32_tc.cu"):
        sizes = re.findall(r"cudaFuncSetAttribute\(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (\w+)\)", source(name))
        assert sizes, name
        for size in sizes:
            assert re.search(r"constexpr int [^;]*\b%s = " % size, source(name)), (name, size)

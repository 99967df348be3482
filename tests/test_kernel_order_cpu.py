"""Orderings inside the kernels that no run can show to be missing (a race that is nearly always won, a wait that is nearly always
short), stated over the kernels' source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "adreno-llms_b200", "csrc")


def source(name):
    """The file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        s = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", s, flags=re.S)


def block_after(s, start):
    """From `start` (a text that occurs once, up to a body's opening brace or before it) to the end of that body."""
    assert s.count(start) == 1, start
    i = s.index("{", s.index(start))
    depth = 0
    for j in range(i, len(s)):
        depth += {"{": 1, "}": -1}.get(s[j], 0)
        if depth == 0:
            return s[i:j + 1]
    raise AssertionError(start)


def test_published_words_are_read_whole():
    """A published word is value and epoch in 64 bits, stored as one; a vector load reads it as one only with 64-bit elements."""
    s = source("decode_plan.cu")
    assert "st.relaxed.gpu.global.u64" in s
    for body in ("bool fetch_piece(", "void poll_batch(", "uint16_t poll_row("):
        loads = re.findall(r"ld\.[a-z0-9_.]+", block_after(s, body)) + re.findall(r"\bld_relaxed_u64\b", block_after(s, body))
        assert loads, body
        assert all(l.endswith("u64") for l in loads), (body, loads)


def test_batched_finish_waits_for_the_reads_of_its_buffer():
    """Where one warp has added up the K parts, it writes its finish layout (8 * NT rows of RED_TS words) over the place of the
    parts it has just read (32 * 8 * NT words each): the lanes meet in between."""
    red_ts = int(re.search(r"constexpr int RED_TS = (\d+);", source("stream_core.cuh")).group(1))
    assert 8 * red_ts > 32 * 8, "the layouts no longer overlap: the meeting is not needed for this"
    _, finish = source("gemv_stream.cu").split("float* const mine = buf + warp * (8 * NT * RED_TS)")
    assert "__syncwarp();" in finish[:finish.index("mine[")]


def test_norm_weight_is_read_after_the_launch_before():
    """nn_rmsnorm takes any buffer as its weight, so also one that the call before has written."""
    body = block_after(source("misc.cu"), "rmsnorm_rows_kernel(const uint16_t* __restrict__ x")
    early = body[:body.index("pdl_wait_prior_grid()")]
    assert not re.search(r"\b(gw|xr|orow)\[", early), early


def test_launches_that_read_ahead_ask_first():
    """The streaming kernel and the GEMM fetch weights (and biases) before they wait for the launch before: each call site has asked
    whether a launch in flight may be writing one."""
    calls = re.findall(r"launch_(?:stream|gemm_tc)\(([^;]*)\);", source("api.cpp"))
    assert len(calls) >= 3
    assert all("c->use_pdl && overlap" in c for c in calls), calls


def test_waits_have_time_for_the_launch_before():
    """Launches begin while the one before them runs, and what they wait for (tokens, or room that the use of tokens frees) comes
    only after it: every limit on such a wait is far above the longest launch, and none is written out by itself."""
    limit = int(re.search(r"constexpr long long WAIT_CYCLES = (\d+)ll;", source("ptx.cuh")).group(1))
    assert limit >= 2 * 1_900_000_000          # two seconds at the highest clock
    for name in ("gemm_tc.cu", "gemv_stream.cu", "ptx.cuh"):
        s = source(name)
        assert not re.search(r"clock64\(\) - t0 [<>] 200000000ll", s) and "limit_cycles = 200000000ll" not in s, name
    ring = block_after(source("decode_plan.cu"), "if (warp == PCW) {")
    assert "oldest == 0u ? WAIT_CYCLES + 4 * P.wait_cycles" in ring


def test_tables_that_any_thread_fills_are_atomic():
    """What a device's properties give is kept in static tables, which calls of any thread read and fill."""
    tables = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cpp", ".h", ".cuh")):
            tables += [(name, t.strip()) for t in re.findall(r"\bstatic ([^;(={]*\bcached\b)", source(name))]
    assert len(tables) >= 2 and all(t.startswith("std::atomic<") for _, t in tables), tables

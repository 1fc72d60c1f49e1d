"""The convolution kernels' whole-warp instructions, read from their source: tcgen05.ld,
alloc and dealloc are .aligned (undefined in a warp that has diverged), and a lane that
leaves a loop on an answer of its own leaves the others waiting in the next vote.

- A loop that issues a TMEM load has no `continue` (lanes that take it would load while the
  others still work), and rejoins the warp after its last per-lane branch.
- TMEM is allocated and released right after a barrier of the warp.
- A loop left because of the abort flag asks the whole warp (warp_any), except in code that
  one elected lane runs.
"""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "offlinerenderer_b200", "csrc",
                   "conv_tc.cu")


def _source():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _close(s, i):
    """Position of the brace that closes the one at i."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == "{") - (s[k] == "}")
        if depth == 0:
            return k
    raise ValueError("unbalanced braces")


def _loops_with(s, call):
    """Bodies of the innermost for loops that contain `call`."""
    out = []
    for m in re.finditer(re.escape(call) + r"\(", s):
        best = None
        for f in re.finditer(r"\bfor \([^{}]*\) \{", s[:m.start()]):
            if _close(s, f.end() - 1) > m.start():
                best = s[f.end():_close(s, f.end() - 1)]
        if best is not None:
            out.append(best)
    return out


def test_no_lane_skips_past_a_tmem_load():
    s = _source()
    loops = _loops_with(s, "tmem_ld16") + _loops_with(s, "tmem_ld32_async")
    assert len(loops) >= 4
    for body in loops:
        assert not re.search(r"\bcontinue;", body), body
        m = re.search(r"tmem_ld(16|32_async)\(", body)
        # what runs from this load to the next one, around the loop
        between = body[m.end():] + body[:m.start()]
        rejoined = between.rfind("__syncwarp();")
        assert not re.search(r"\bif \((?!plain|sliceC)", between[max(rejoined, 0):]), body


def test_tmem_is_allocated_and_released_by_whole_warps():
    s = _source()
    for name in ("tmem_alloc", "tmem_dealloc"):
        uses = list(re.finditer(name + r"\(", s))
        assert len(uses) == 2
        for m in uses:
            before = [x.strip() for x in s[:m.start()].split("\n")[-4:]]
            # the warp that allocates in k_conv_wgrad has not branched since the launch
            joined = any("__syncwarp();" in x or "__syncthreads();" in x for x in before)
            assert joined or (name == "tmem_alloc" and "if (warp == 1) {" in before), before


def test_the_abort_flag_is_read_by_the_whole_warp():
    s = _source()
    for m in re.finditer(r"\*abortFlag\b(?! =)", s):
        line = s[s.rfind("\n", 0, m.start()) + 1:s.find("\n", m.start())].strip()
        one_lane = line.startswith(("ok = ok && !*abortFlag", "if (*abortFlag) {", "if (threadIdx.x == 0 &&"))
        assert "warp_any(*abortFlag)" in line or one_lane, line

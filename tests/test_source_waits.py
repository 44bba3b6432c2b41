"""Read from the kernels' source: how threads that share barriers leave when a wait runs out."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fastkernels_b200" / "csrc"


def _branch(text, start):
    """The text of the braces that open after `start`."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name,mark", [("fk_gemm.cu", "} else if (warp >= 2) {"),
                                       ("fk_block.cu", "    const int t128 = threadIdx.x - 64;")])
def test_epilogue_threads_of_few_row_products_leave_together(name, mark):
    """128 threads meet at named barriers, and each waits for the accumulators by itself: one that
    left alone when its wait ran out would leave the others there without end.  So no thread's own
    wait, nor what it reads of the abort flag, decides about a loop or a barrier."""
    text = _code(name)
    start = text.index(mark) if mark.startswith("}") else text.rindex("{", 0, text.index(mark))
    body = _branch(text, start)
    assert "named_bar_sync(1, 128)" in body
    assert len(re.findall(r"\(void\)gemm_wait\(&acc_full", body)) == 1
    assert "gemm_wait(" not in body.replace("(void)gemm_wait(&acc_full", "")
    # who leaves, and by what: a chunk that is not there, one thread's wait for flags, and a
    # decision that one thread wrote ahead of a barrier
    leaves = re.findall(r"([^;{}]*)\b(?:break|return)\b", body)
    allowed = {"if (c >= p.m)", "if (*stop)"} | \
        {x for x in leaves if "atomicOr(p.status" in x}
    assert {x.strip() for x in leaves if x.strip()} <= allowed
    for cond in re.findall(r"(?:while|for) \(([^{}]*)\) \{", body):
        assert "ok" not in re.findall(r"\w+", cond)
    for m in re.finditer(r"if \(([^{};]*abort_flag[^{};]*)\)\s*(\{)?", body):
        after = _branch(body, m.end() - 1) if m.group(2) else body[m.end():body.index(";", m.end())]
        assert "bar_sync" not in after


def test_register_splits_are_checked_before_the_launch():
    """setmaxnreg.inc waits without end where a CTA was launched with fewer registers than its
    split adds up to.  Each kernel that has it names its split, and its launch asks the compiled
    kernel for its registers and refuses."""
    have = [f.name for f in sorted(CSRC.glob("*.cu*")) if "setmaxnreg.inc" in _code(f.name)]
    assert have == ["fk_plain.cu", "fk_prefill.cu"]
    for name in have:
        text = _code(name)
        # no number in the instruction itself
        assert re.findall(r'setmaxnreg\.(?:inc|dec)\.sync\.aligned\.u32 ([^;]*);', text) == ["%0"] * \
            len(re.findall("setmaxnreg", text))
        needed = re.search(r"(\w*REGS_?NEEDED) =", text, re.I).group(1)
        assert re.search(r"FK_REQUIRE\(launch_regs \* [\w:]+ >= (?:Tile::)?%s," % needed, text)
        assert "cudaFuncGetAttributes(&f, " in text and "f.numRegs" in text


def _headers(text, at):
    """What stands before each brace that is open at `at`, and before the statement itself."""
    out, depth, i, end = [], 0, at, at
    while i > 0:
        i -= 1
        if text[i] == "}":
            depth += 1
        elif text[i] == "{":
            if depth == 0:
                j = max(text.rfind(c, 0, i) for c in ";{}")
                out.append(text[j + 1:i])
            else:
                depth -= 1
    j = max(text.rfind(c, 0, end) for c in ";{}")
    return out + [text[j + 1:end]]


@pytest.mark.parametrize("name", sorted(f.name for f in CSRC.glob("*.cu*")))
def test_warps_leave_their_waits_together(name):
    """Lanes may see a barrier's phase one by one, and matrix instructions, tensor-memory accesses and
    named barriers want whole warps: a wait of more than one lane goes through a form that gives all
    lanes one answer (*_wait_warp, a vote), or is followed by __syncwarp()."""
    text = _code(name)
    for m in re.finditer(r"\b(?:pf|gl|gg|att|gemm|mbar)_wait\(", text):
        heads = _headers(text, m.start())
        line = heads[-1]
        if "__device__" in line or "__all_sync(" in line or "gt_all(" in line:
            continue
        one = re.compile(r"lane == 0|threadIdx\.x == (?:0|64)|t128 == 0|feeds")
        if any(one.search(h) for h in heads):
            continue
        rest = text[m.start():]
        assert re.match(r"[^;]*;\s*(?:__syncwarp\(\);|return __all_sync\()", rest), rest[:200]
    for m in re.finditer(r'"bar\.(?:sync|arrive) ', text):
        assert text[:m.start()].rstrip().endswith("__syncwarp();\n  asm volatile(".strip()) or \
            "__syncwarp();" in text[max(0, m.start() - 60):m.start()]


def test_decode_attention_leaves_with_all_its_warps():
    """Eight warps meet at named barriers when an item's keys are through: one leaves its loop at the
    end marker, or where att_give_up says that all of them have given up."""
    text = _code("fk_attn.cu")
    body = _branch(text, text.index("for (;;) {", text.index("attn_decode_kernel(")))
    assert "named_bar_sync(1, ATT_NW * 32)" in body and "return" not in body
    leaves = [" ".join(x.split()) for x in re.findall(r"([^;{}]*)\bbreak\b", body)]
    assert leaves == ["if (!att_wait_warp(&full[stage], phase, abort_flag, p.status) && "
                      "att_give_up(&full[stage], phase, quit))", "if (meta.flags & TILE_END)"]


@pytest.mark.parametrize("seed", range(40))
def test_giving_up_is_one_decision(seed):
    """att_give_up step by step, in any order of its atomic steps: either all eight warps leave, or
    every one whose tile comes goes on, and none waits for ever."""
    import random
    rng = random.Random(seed)
    closed, warps = 1 << 16, 8
    state = {"quit": 0, "tile": False, "comes": rng.random() < 0.7}

    def warp():
        if state["tile"] and rng.random() < 0.5:
            return False                        # its own wait saw the tile
        seen = state["quit"]
        yield
        while True:
            old = state["quit"]
            if old == seen:
                state["quit"] = closed if seen + 1 == warps else seen + 1
            yield
            if old == seen:
                break
            seen = old
        while True:
            yield
            if state["quit"] & closed:
                return True
            if not state["tile"]:
                continue
            seen = state["quit"]
            yield
            while not seen & closed:
                old = state["quit"]
                if old == seen:
                    state["quit"] = seen - 1
                yield
                if old == seen:
                    break
                seen = old
            return bool(seen & closed)
    running, left = [warp() for _ in range(warps)], []
    for step in range(20000):
        if not running:
            break
        if state["comes"] and rng.random() < 0.02:
            state["tile"] = True
        w = rng.choice(running)
        try:
            next(w)
        except StopIteration as e:
            running.remove(w)
            left.append(e.value)
            if e.value is False:
                assert state["tile"]
    assert not running and len(set(left)) == 1

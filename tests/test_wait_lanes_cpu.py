"""Waits of the kernel's whole-warp roles, read from the source: a lane that gives up on its own must not leave the others of its
warp at an operation that needs all of them. So a wait made lane by lane runs in one lane, or sets the flag of a role without such
operations (gather), or its answer is voted on before anything is skipped (epilogue)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "unimonomoe_b200", "csrc")


def _code(name):
    return [re.sub(r"//.*", "", line) for line in open(os.path.join(CSRC, name))]


def _enclosing(lines, at):
    """The lines that open the blocks around line `at`, innermost first."""
    depth = 0
    for i in range(at, -1, -1):
        for ch in reversed(lines[i] if i < at else ""):
            if ch == "}":
                depth += 1
            elif ch == "{":
                if depth == 0:
                    yield lines[i]
                else:
                    depth -= 1


def test_lane_by_lane_waits():
    wrong = []
    for name in ("mono_kernel.cu", "slot_copies.cuh"):
        lines = _code(name)
        for i, line in enumerate(lines):
            if not re.search(r"\bmbar_wait\(", line) or "return mbar_wait(" in line:   # (the MMA warp's choice: below)
                continue
            flag = re.search(r"if \(.*!dead && !mbar_wait\(.*\)\) dead = true;|if \(!dead\) given_up = !mbar_wait\(", line)
            if not flag and not any("lane == 0" in b for b in _enclosing(lines, i)):
                wrong.append(f"{name}:{i + 1}: {line.strip()}")
    assert not wrong, wrong


def test_what_skips_a_read_out_is_voted_on():
    """tcgen05.ld and the __syncwarp behind it: by every lane of a warp or by none."""
    text = "".join(_code("mono_kernel.cu"))
    split = text[text.index("void split_phase("):text.index("void __launch_bounds__(BLOCK, 1) moe_prefill_kernel(")]
    split = split[split.index("auto down_col"):]
    assert re.search(r"dead = __any_sync\(0xFFFFFFFFu, dead\);\s*return buf;", split) and split.count("dead = true;") == 2   # and `meet`: the whole role
    epilogue = text[text.index("bool dead = false, given_up = false;"):text.index("if constexpr (REST) {", text.index("given_up"))]
    assert "dead = true" not in epilogue and epilogue.count("dead = __any_sync(0xFFFFFFFFu, given_up);") == 2


def test_mma_warp_waits_together():
    text = "".join(_code("mono_kernel.cu"))
    assert re.search(r"if constexpr \(MONO_MMA_WARP != 0\) return mbar_wait_warp\(bar, parity, wc, site\);", text)


def test_announced_copies_are_waited_for():
    """Every ring that copies are announced on is drained by the role that announced them, but for the weights of the expert phase,
    behind which an aborting CTA pauses; and the pause is one that lasts."""
    for name, weights in (("mono_kernel.cu", {"S.fullB", "S.sp.fullB"}), ("slot_copies.cuh", set())):
        text = "".join(_code(name))
        announced = set(re.findall(r"mbar_arrive_expect_tx\(&([\w.]+)\[", text))
        drained = set(re.findall(r"drain_copies\(([\w.]+),", text))
        assert announced - weights and announced - weights == drained, (name, announced ^ drained)
        assert "__nanosleep" not in text and text.count("if (aborted(ws)) settle();") == (1 if weights else 0)

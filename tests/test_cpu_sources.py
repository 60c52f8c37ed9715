"""What the kernel sources have to keep to and no run can show: what happens after a wait has run out, and what needs a whole warp."""
import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "ml_b200" / "csrc" / "kernels"


def _kernels():
    """(file, name, body without comments, line breaks kept) of every __global__ function."""
    for path in sorted(list(KERNELS.glob("*.cu")) + list(KERNELS.glob("*.cuh"))):
        text = re.sub(r"/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group(0)), path.read_text(), flags=re.S)
        text = re.sub(r"//[^\n]*", "", text)
        for m in re.finditer(r"__global__\s+void[^;{]*?\b(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield path.name, m.group(1), text[m.start():i], text.count("\n", 0, m.start()) + 1


def _heads(body, at):
    """The statement that position `at` is in up to there, and the heads of the blocks around it, innermost first."""
    i = at
    while i > 0:
        end, parens = i, 0
        while i > 0:
            c = body[i - 1]
            parens += {")": 1, "(": -1}.get(c, 0)
            if parens <= 0 and c in "{};":
                break
            i -= 1
        yield body[i:end]
        depth = 0      # to the brace that opens the block around
        while i > 0:
            i -= 1
            depth += {"}": 1, "{": -1}.get(body[i], 0)
            if depth < 0:
                break


def test_the_kernels_are_found():
    names = {name for _, name, _, _ in _kernels()}
    assert {"attn_bwd_q128_k", "attn_bwd_kv128_k", "attn_bwd_fused_tc_kernel", "attn_fwd_rows_tc_kernel", "attn_split_bwd_k", "gemm_tc_kernel"} <= names


def test_a_block_that_has_given_up_stores_no_tile():
    """After a wait has run out, what stands in tensor and shared memory is nobody's result: each tile that leaves asks for the block's word first."""
    found, unasked = 0, []
    for file, name, body, line in _kernels():
        if "s_abort" not in body:
            continue
        for m in re.finditer(r"\btc::tma_store_2d\(|\btile128_rows\(", body):
            found += 1
            if not any("*s_abort" in head for head in _heads(body, m.start())):
                unasked.append(f"{file}:{line + body.count(chr(10), 0, m.start())} {name}")
    assert found >= 7 and not unasked, unasked


ONE_THREAD = re.compile(r"lane == 0|tid == 0|threadIdx\.x == 0|elect_one\(\)|\bleader\(\)|\bloader\(\)|auto issue_\w+ = \[&\]")
WAIT = re.compile(r"(?<!\w)(?:tc::)?(?:wait|mbar_wait)\(")


def _close(body, at):
    """Position behind the parenthesis that closes the one before `at`."""
    depth = 1
    while depth:
        depth += {"(": 1, ")": -1}.get(body[at], 0)
        at += 1
    return at


def test_a_warp_is_together_again_behind_its_waits():
    """A wait is a loop that lanes can leave in different rounds, and tensor-memory accesses, matrix stores and named barriers take a whole warp: behind the
    last wait of a row the warp is brought together before anything else.  Where the answer decides, the lanes have one answer."""
    found, apart = 0, []
    for file, name, body, line in _kernels():
        if "mbar_wait" not in body:
            continue
        for m in WAIT.finditer(body):
            heads = list(_heads(body, m.start()))
            if "auto wait" in heads[0] or any(ONE_THREAD.search(h) for h in heads):
                continue
            found += 1
            end = _close(body, m.end())
            where = f"{file}:{line + body.count(chr(10), 0, m.start())} {name}"
            if body[end] != ";":      # its answer is asked for
                if not heads[0].rstrip().endswith("__all_sync(0xffffffffu,"):
                    apart.append(where)
                continue
            rest = body[end + 1:].lstrip()
            if not re.match(r"__syncwarp\(\)|__syncthreads\(\)|(?:if \([^;{}]*\) )?wait\(|(?:tc::tc_fence_after\(\);\s*)?if \(__all_sync\(", rest):
                apart.append(where)
    assert found > 20 and not apart, "\n".join(apart)


def test_a_block_that_gives_up_leaves_a_number():
    """The word that says so is the number of the wait that ran out: a wait numbered 0 would run out unseen."""
    numbers = [body[m.end():_close(body, m.end()) - 1].rsplit(",", 1)[1].strip()
               for _, _, body, _ in _kernels() if "s_abort" in body for m in re.finditer(r"(?<![\w:])wait\(", body)]
    assert len(numbers) > 90 and all(n == "where" or re.search(r"[1-9]", n) for n in numbers)


def test_every_refused_index_has_its_words():
    from ml_b200.ops.native import describe_error
    details = {int(d, 16) for path in KERNELS.glob("*.cu*") for d in re.findall(r"MLB_ERR_BOUNDS, (0x[0-9A-Fa-f]+)\)", path.read_text())}
    assert 0xE1 in details
    assert not [hex(d) for d in details if describe_error(3 << 24 | d).endswith(f"detail {d:#x}")]

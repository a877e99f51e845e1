"""What can be told of the native sources without compiling them or a GPU."""
import collections
import re


def test_every_exported_function_is_defined_once():
    """The library is linked from every source under the kernel folders: a second file with the same functions stops the link."""
    from openagents_b200 import _build
    for sources in (_build.cuda_sources(), _build.host_sources()):
        defined = collections.defaultdict(list)
        for path in sources:
            text = re.sub(r"//[^\n]*", "", path.read_text())
            for m in re.finditer(r"(?:B200_API|extern \"C\")[^;{}()]*?\b(b200_\w+)\s*\([^;{}]*\)\s*\{", text):
                defined[m.group(1)].append(path.name)
        assert len(defined) > 20
        assert {name: files for name, files in defined.items() if len(files) > 1} == {}


def _stale_read(ring, operands, slot_first, stages=9):
    """Walk every interleaving of the fused-dequant GEMM's hand-over: loads that land in any order, two groups of expansion warps that take stages in
    turn, MMAs that finish in order.  A wait passes when the barrier's phase has the other parity, as ``mbarrier.try_wait.parity`` does.  Returns a
    stage whose bytes a group reads before they have landed, or None."""
    # (loads issued, loads landed, per group (its stage, step), per stage whether released / expanded, MMAs finished)
    start = (0, frozenset(), ((0, 0), (1, 0)), frozenset(), frozenset(), 0)
    seen, todo = {start}, [start]
    turn = lambda g, n: (g // n) & 1

    def phases(done, g, n):                                        # completed phases of the barrier of stage g's slot
        return sum(s % n == g % n for s in done)

    while todo:
        issued, landed, groups, released, expanded, finished = todo.pop()
        mma = range(finished)
        after = []
        if issued < stages and (phases(released, issued, ring) & 1) != (turn(issued, ring) ^ 1):
            after.append((issued + 1, landed, groups, released, expanded, finished))
        for g in range(issued):
            if g not in landed:
                after.append((issued, landed | {g}, groups, released, expanded, finished))
        if finished in expanded:
            after.append((issued, landed, groups, released, expanded, finished + 1))
        for i, (g, step) in enumerate(groups):
            if g >= stages:
                continue
            steps = ("slot", "bytes", "finish") if slot_first else ("bytes", "slot", "finish")
            if steps[step] == "slot" and (phases(mma, g, operands) & 1) == (turn(g, operands) ^ 1):
                continue
            if steps[step] == "bytes":
                if (phases(landed, g, ring) & 1) == turn(g, ring):
                    continue
                if g not in landed:
                    return g
            nxt = (g + 2, 0) if step == 2 else (g, step + 1)
            g2 = tuple(nxt if j == i else x for j, x in enumerate(groups))
            if steps[step] == "finish":
                after.append((issued, landed, g2, released | {g}, expanded | {g}, finished))
            else:
                after.append((issued, landed, g2, released, expanded, finished))
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_fused_dequant_gemm_reads_no_stage_before_it_has_landed():
    from openagents_b200 import _build
    text = (_build.CSRC / "kernels" / "qgemm_tc05.cu").read_text()
    rings = [int(v) for v in re.search(r"RS = WT == QW_Q4KR \? \(QBN == 64 \? (\d+) : (\d+)\) : \(QBN == 64 \? (\d+) : (\d+)\)", text).groups()]
    operands = [int(v) for v in re.search(r"kAS = QBN == 64 \? (\d+) : (\d+)", text).groups()] * 2
    rule = "kSlotFirst = RS % kDqGroups != 0 && RS < kAS + 3" in text
    for ring, ops in zip(rings, operands):
        assert _stale_read(ring, ops, rule and ring % 2 != 0 and ring < ops + 3) is None, (ring, ops)
    # the walk does find such a read: an odd ring of three, with the bytes waited for first
    assert _stale_read(3, 2, False) is not None and _stale_read(3, 2, True) is None

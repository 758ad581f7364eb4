"""Kernels launched to start before their predecessors end (launch_dependent):
what a predecessor writes is not read through the read-only path, whose data
must not change while the kernel runs, and the kernel runs from before its
predecessor's end.  A misread needs a stale line in the right L1, so the rule
is held on the source."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "graphwalker_b200" / "csrc"
# what was copied up, or built, before the first kernel of the call
UPLOADED = {"seg_first"}


def _sources() -> dict[str, str]:
    return {f.name: re.sub(r"//[^\n]*", "", f.read_text()) for f in sorted(CSRC.glob("*.cu*"))}


def _kernels(text: str) -> dict[str, tuple[str, str]]:
    """name -> (parameters, body) of every __global__ function of a source."""
    found = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?(\w+)\(", text):
        end, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        at = text.index("{", end)
        stop, depth = at + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[stop], 0)
            stop += 1
        found[m.group(1)] = text[m.end():end - 1], text[at:stop]
    return found


def test_dependent_kernels_do_not_read_predecessors_through_the_read_only_path():
    seen = {}
    for name, text in _sources().items():
        waiting = {k: v for k, v in _kernels(text).items() if "wait_for_previous()" in v[1]}
        seen.update(waiting)
        for kernel, (parameters, _) in waiting.items():
            for p in parameters.split(","):
                if "const" in p and "__restrict__" in p:
                    assert p.split()[-1] in UPLOADED, f"{name}: {kernel}: {p.strip()}"
    assert {"partition_scan_kernel", "partition_scatter_kernel", "walk_query_kernel", "topk_few_kernel"} <= set(seen)


def test_dependent_kernels_read_tables_and_lists_coherently():
    text = _sources()["gw_ppr.cu"]
    for reader, load in (("LiveSlotKey : SlotKey", "load_slot"), ("LiveCandKey : CandKey", "__ldcg")):
        fetch = re.search(rf"struct {reader} \{{.*?fetch\(uint32_t i\) const \{{ return (\w+)\(", text, re.S)
        assert fetch.group(1) == load, f"{reader}::fetch reads with {fetch.group(1)}"
    few = _kernels(text)["topk_few_kernel"][1]
    assert "LiveSlotKey{table_slots(" in few and few.count("table_slots(") == 1
    assert "LiveCandKey{{seg_cand" in few and few.count("CandKey{") == 1
    slot = re.search(r"load_slot\(.*?\n\}", text, re.S).group(0)
    assert "ld.relaxed.gpu.global" in slot and ".nc" not in slot


def test_what_a_scan_reads_and_writes_shares_no_line():
    """The pool table's arrays start on lines of their own."""
    header = re.sub(r"//[^\n]*", "", (CSRC / "gw_internal.h").read_text())
    stride = re.search(r"static size_t stride\(uint32_t nbuckets\) \{ return (.*?); \}", header).group(1)
    for nb in (1, 15, 16, 17, 33, 7999):
        n = eval(stride.replace("(size_t)nbuckets", str(nb)).replace("/", "//"))
        assert nb <= n < nb + 16 and n * 8 % 128 == 0
    engine = _sources()["gw_engine.cu"]
    assert "entries = PoolTable::stride(nb)" in engine
    for array in ("table.n + entries", "table.cap + entries", "table.place + entries"):
        assert array in engine

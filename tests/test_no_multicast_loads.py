"""No TMA or bulk load of the library carries the cluster multicast qualifier: the same library serves tensor-parallel ranks,
whose operands may lie in a peer's memory. (tcgen05.commit may: it is an arrival on barriers, not a load.)"""
import pathlib
import re

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_no_bulk_load_with_cluster_multicast():
    found = []
    for path in sorted((ROOT / "llm-inference_b200").rglob("*.c*")) + sorted((ROOT / "tools").rglob("*.cu")):
        for m in re.finditer(r"cp\.async\.bulk[^;\[]*", re.sub(r'"\s*"', "", path.read_text(errors="replace"))):
            if "multicast" in m.group(0):
                found.append(f"{path.relative_to(ROOT)}: {m.group(0)[:120]}")
    assert not found, found

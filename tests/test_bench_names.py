"""The stages and kernels that bench.py reports are the ones the engine has (CPU)."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SOURCES = "".join(p.read_text() for p in sorted((ROOT / "pm7-rs_b200" / "csrc").glob("*.cu")))
STAGES = set(re.findall(r"\bStage \w+\(\w+, \"(\w+)\"\)", SOURCES))


def test_every_stage_bench_reads_is_timed_by_the_engine():
    asked = set(re.findall(r"prof\.get\(\"(\w+)\"", (ROOT / "bench.py").read_text()))
    assert asked and not asked - STAGES, asked - STAGES


def test_every_traffic_line_names_a_stage():
    lines = (ROOT / "profiles" / "traffic.txt").read_text().splitlines()
    names = {ln.split()[0] for ln in lines if ln.strip() and not ln.startswith("#")}
    assert names and not names - STAGES, names - STAGES


def test_every_kernel_bench_names_exists():
    named = set(re.findall(r"\bk_[a-z0-9_]+", (ROOT / "bench.py").read_text()))
    defined = set(re.findall(r"\b(k_[a-z0-9_]+)\s*\(", SOURCES))
    assert named and not named - defined, named - defined


def test_traffic_is_given_at_the_order_it_was_captured_at():
    import bench

    assert bench.read_traffic("fock", bench.TRAFFIC_NAO) > 0
    assert bench.read_traffic("fock", 6000) is None

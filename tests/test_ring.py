"""What a kernel waits for before it ends after a wait that gave up: the copies that are still on their way into its shared memory.
Read and simulated on the CPU; no kernel is made to give up here."""
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "lumen_b200" / "csrc"


def test_drain_waits_exactly_for_the_copies_in_flight(tmp_path):
    out = tmp_path / "ring_check"
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", str(CSRC), str(ROOT / "tests" / "cpp" / "ring_check.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_no_wait_for_either_parity():
    """One of the two parities of an mbarrier always tests as complete, so a loop that ends with either of them never waits."""
    either = re.compile(r"bar_try\(([^;]*?), 0\)\s*&&\s*!\s*\w*bar_try\(\1, 1\)")
    bad = [f"{p.name}: {m.group(0)}" for p in sorted(CSRC.glob("*.cu*")) for m in either.finditer(p.read_text())]
    assert not bad, bad

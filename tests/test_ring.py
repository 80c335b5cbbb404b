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


def test_answers_of_bounded_waits_are_agreed_on():
    """Threads of a CTA may see a wait end differently near its limit; where whole warps or the CTA meet again behind it, they take one answer."""
    for name in ("gemm_rows.cu", "gemm_tc.cu"):
        text = (CSRC / name).read_text()
        assert len(re.findall(r"const bool have = bar_wait\(&done", text)) == len(re.findall(r"__syncthreads_and\(have\)", text)) == 1, name
        assert not re.search(r"\bhave && ", text), name
    waits = re.findall(r"alive = (.*)bar_wait", (CSRC / "attention.cu").read_text() + (CSRC / "attn_rows.cu").read_text())
    assert len(waits) == 3 and all("__all_sync" in w for w in waits), waits


def test_limits_start_behind_the_kernel_before():
    """Kernels that start early count their bounded waits from the end of their predecessor: no wait on a barrier before pdl_wait()."""
    for name in ("gemm_rows.cu", "attn_rows.cu"):
        text = (CSRC / name).read_text()
        body = text[text.index("    pdl_launch();"):]
        branches = re.split(r"\n    \} else if \(", body[: body.index("bar_wait(&done") if "bar_wait(&done" in body else len(body)])
        for b in branches:
            if "bar_wait(" in b:
                assert "pdl_wait()" in b[: b.index("bar_wait(")], (name, b[:60])


def test_dependents_start_behind_the_allocation():
    """A kernel launched behind one that takes tensor memory may take some before it waits: every CTA of the first has its own by the time it lets
    dependents start, or the two could wait for one another without a limit."""
    seen = 0
    for p in sorted(CSRC.glob("*.cu")):
        for body in p.read_text().split("__global__")[1:]:
            if "tcgen05.alloc" in body and "pdl_launch();" in body:
                between = body[body.index("tcgen05.alloc"): max(body.index("tcgen05.alloc"), body.index("pdl_launch();"))]
                assert "tcgen05.relinquish_alloc_permit" in between and "__syncthreads()" in between, p.name
                seen += 1
    assert seen == 3


def test_peer_addresses_come_from_mapa():
    """Where the window of a cluster's other CTA lies is the machine's business: addresses in it come from mapa, not from masked bits."""
    for p in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"0xF[0-9A-Fa-f]FFFFFF|kPeerMask", p.read_text()), p.name
    assert "mapa.shared::cluster" in (CSRC / "gemm_pair.cu").read_text()


def test_tensor_memory_is_kept_until_the_mmas_end():
    """Every kernel that gives tensor memory back waits, after a wait that gave up, for a barrier that its last MMAs arrive at."""
    for p in sorted(CSRC.glob("*.cu")):
        text = p.read_text()
        waits = re.findall(r"drain_mmas\(&\w+\)|drain_ring\(&(?:done|quiet), 1, 1\)", text)
        assert text.count("tcgen05.dealloc") == len(waits), p.name

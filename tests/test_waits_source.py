"""Every spin-wait of the kernels is one of the bounded functions of waits.cuh, and the self-test drives each kind."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "fluidlets_gb300" / "csrc"


def code(p):
    return re.sub(r"//.*", "", p.read_text())


def test_waits_live_in_one_file():
    for p in sorted(CSRC.glob("*.cu*")):
        if p.name != "waits.cuh":
            assert "try_wait" not in code(p), p.name
            assert "global_ns(" not in code(p), p.name  # a loop with a limit of its own


def test_the_self_test_calls_every_kind():
    kinds = set(re.findall(r"__forceinline__ bool (\w+)\(", code(CSRC / "waits.cuh")))
    kinds -= {"mbar_try_wait", "cluster_try_wait"}  # single probes
    called = code(CSRC / "waits.cu")
    # (mbar_drain is mbar_wait without the early end on another's failure)
    assert {"wait_published4", "wait_parity", "grid_sync", "mbar_wait", "cluster_wait"} <= kinds
    for k in kinds - {"mbar_drain"}:
        assert re.search(rf"\b{k}\(", called), k


def test_limits_are_passed_to_every_wait():
    for p in sorted(CSRC.glob("*.cu")):
        for m in re.finditer(r"\b(cluster_wait|mbar_wait|mbar_drain|wait_parity|wait_published4)\(", code(p)):
            call = code(p)[m.start():m.start() + 200].split(";")[0]
            assert "kWaitLimitNs" in call or "limit_ns" in call, (p.name, call)

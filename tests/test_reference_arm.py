"""bench.py --impl reference where the reference's own harness is missing: the line says that its
value is not the reference's."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_port_is_not_passed_off_as_the_reference():
    import oracle as O
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"], cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout.strip().splitlines()[-1])
    assert d["impl"] == "reference"
    assert ("unavailable" in d) == (not O.ref_available())
    assert (d["cpu_baseline"]["kind"] == "reference") == O.ref_available()

"""The bench's reference arm runs the reference's own code or says that it cannot:
never the oracle's restatement, which is this repository's."""

import json
import pathlib
import subprocess
import sys

from native import have_ref

ROOT = pathlib.Path(__file__).resolve().parent.parent


def test_reference_arm_is_the_reference_or_unavailable():
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--n",
                          "2000", "--steps", "1", "--warmup", "3"], check=True,
                         capture_output=True, text=True).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["impl"] == "reference"
    assert ("unavailable" in line) != have_ref()
    if have_ref():
        assert line["cpu_baseline"]["kind"] == "reference"

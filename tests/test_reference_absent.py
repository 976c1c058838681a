"""Without the reference library a comparison with it is skipped, not failed,
so that a run that stops at the first failure goes on."""
import subprocess
import sys

from conftest import ROOT

CASE = """
import oracle
from pathlib import Path

def test_compares():
    oracle.REF_SO = Path("/nonexistent/libmlods_ref.so")
    oracle._ref = None
    oracle.ref()
"""


def test_comparison_is_skipped(tmp_path):
    (tmp_path / "test_case.py").write_text(CASE)
    res = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider", str(tmp_path)], cwd=ROOT,
                         env={"PYTHONPATH": str(ROOT), "PATH": "/usr/bin:/bin"}, capture_output=True, text=True,
                         timeout=120)
    assert res.returncode == 0 and "1 skipped" in res.stdout, res.stdout + res.stderr

"""Tests that call a tool built from the reference's sources, where it is absent."""
import os
import subprocess
import sys

from conftest import ROOT

CASES = """
import os, subprocess
from conftest import TOOLS
def test_absent_tool():
    subprocess.run([os.path.join(TOOLS, "no_such_tool")], check=True)
def test_other_missing_file():
    open(os.path.join(os.path.dirname(__file__), "no_such_file"))
def test_failing_before_the_tool():
    assert not TOOLS
    subprocess.run([os.path.join(TOOLS, "no_such_tool")], check=True)
def test_after():
    pass
"""


def test_an_absent_tool_skips_its_test_and_nothing_else(tmp_path):
    (tmp_path / "test_cases.py").write_text(CASES)
    p = subprocess.run([sys.executable, "-m", "pytest", "-v", "-p", "conftest", "--rootdir", str(tmp_path),
                        "--noconftest", str(tmp_path)], capture_output=True, text=True, cwd=tmp_path,
                       env=dict(os.environ, PYTHONPATH=os.path.join(ROOT, "tests")))
    got = {line.split("::")[1].split()[0]: line.split("::")[1].split()[1] for line in p.stdout.splitlines()
           if line.startswith("test_cases.py::")}
    assert got == dict(test_absent_tool="SKIPPED", test_other_missing_file="FAILED",
                       test_failing_before_the_tool="FAILED", test_after="PASSED"), p.stdout[-3000:] + p.stderr[-2000:]

"""Runs a piece of test code in a process of its own, where nothing has been tuned or pinned yet."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))


def run_fresh(code: str) -> None:
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(HERE), HERE]))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-4000:]

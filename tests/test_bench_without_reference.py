"""bench.py where the reference's libraries (oracle/_ref) were not built: the
CPU baseline is the restatement alone, and the reference arm prints one line
that says it is unavailable."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = ("import sys; sys.argv = ['bench.py']; sys.path.insert(0, %r); import bench; from oracle import oracle as O; "
         "O.timing_build = lambda base: ('/nonexistent/' + base + '.so', ''); "
         "full = bench.cpu_baseline; "
         "bench.cpu_baseline = lambda steps=2, one_rank_steps=2: full(steps, one_rank_steps, level=2); " % ROOT)


def run(code):
    env = {k: v for k, v in os.environ.items() if k != "RANK"}
    out = subprocess.run([sys.executable, "-c", SETUP + code], cwd=ROOT, env=env, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return [json.loads(line) for line in out.stdout.splitlines() if line.strip()]


def test_cpu_baseline_is_the_restatement():
    cb, = run("import json; print(json.dumps(bench.cpu_baseline()))")
    assert cb["kind"] == "port" and cb["cores"] == 1 and cb["value"] > 0 and "not built" in cb["sample"]


def test_reference_arm_says_that_it_is_unavailable():
    line, = run("import argparse; bench.run_reference(argparse.Namespace(steps=2, warmup=3))")
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
    assert line["cpu_baseline"]["kind"] == "port"

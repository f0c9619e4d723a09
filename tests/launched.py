"""Kernels that a piece of code launches, as torch's profiler sees them."""
import json
import os
import subprocess
import sys
import textwrap

from conftest import ROOT

PROLOGUE = """
import json, os, sys, tempfile
import torch
from torch.profiler import ProfilerActivity, profile
import meikey_b200 as mk
torch.cuda.init()
with profile(activities=[ProfilerActivity.CUDA]) as prof:
{body}
    torch.cuda.synchronize()
path = os.path.join(tempfile.mkdtemp(), "trace.json")
prof.export_chrome_trace(path)
events = json.load(open(path))["traceEvents"]
print("KERNELS " + json.dumps([[e["name"], e["args"]] for e in events if e.get("cat") == "kernel"]))
"""


def kernels_of(body: str):
    """[(kernel name, launch attributes)] of `body` (statements using `mk`), run in a process of its own."""
    code = PROLOGUE.format(body=textwrap.indent(textwrap.dedent(body).strip(), "    "))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.environ.get("PYTHONPATH", "")]))
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env, cwd=ROOT)
    assert run.returncode == 0, run.stderr
    line = next(x for x in run.stdout.splitlines() if x.startswith("KERNELS "))
    return [tuple(k) for k in json.loads(line[len("KERNELS "):])]

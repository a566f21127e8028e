"""A process that may not start enough threads: submitting a job reports it, and works once it may."""
import os
import subprocess
import sys

import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(180)]

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, sys
import gianduia_b200 as G
from gianduia_b200 import scenes
left = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "gnd_test_threads")
ctx = G.GpuContext(0)
sid = ctx.upload(G.HostScene.load_xml(scenes.cornell(sys.argv[2], width=16, height=16, spp=1)))
for n in (0, 1):
    left.value = n
    try:
        ctx.submit(sid)
        sys.exit("a job was accepted without threads to serve it")
    except G.GndError:
        pass
left.value = -1
film, st = ctx.wait(ctx.submit(sid), timeout_ms=20000)
assert st["state"] == "done"
ctx.close()
print("served")
"""


def test_submit_without_threads(tmp_path):
    lib = str(tmp_path / "libfew_threads.so")
    subprocess.run(["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-O1", "-shared", "-fPIC",
                    os.path.join(ROOT, "tests", "cpp", "few_threads.cpp"), "-ldl", "-o", lib], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", PROGRAM, lib, str(tmp_path)], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "served", r.stderr[-2000:]

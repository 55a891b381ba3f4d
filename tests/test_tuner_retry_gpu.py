"""A step whose timing found no memory for its scratch is timed by a later call."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# 512 x 512 x 128: a spectrum of 135 MB, a z convolution's scratch twice that
CODE = r"""
import json, os
import numpy as np, torch
from petakit5d_b200 import _lib, synth
from petakit5d_b200 import decon as D

shape = (512, 512, 128)
psf = synth.gaussian_psf((9, 9, 9), 1.2, 2.0)
psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1])
d_in = torch.randint(90, 900, shape[::-1], dtype=torch.int16, device="cuda")
out = torch.empty(shape[::-1], dtype=torch.float32, device="cuda")
ctx = _lib.Context(0)

def run():
    D.decon_device("omw", d_in, "uint16", shape, psf, psf_b, 1, ctx=ctx, out=out, Background=100, save16bit=False)
    torch.cuda.synchronize()
    return len(ctx.tune_read())

os.environ["PK_TUNE"] = "0"          # buffers, OTFs and kernels first
run(); run()
del os.environ["PK_TUNE"]
free = torch.cuda.mem_get_info()[0]
block = torch.empty(free - (96 << 20), dtype=torch.uint8, device="cuda")
tight = [run() for _ in range(2)]
ref = out.cpu()
del block
torch.cuda.empty_cache()
later = run()
print(json.dumps({"tight": tight, "later": later, "sources": [t["source"] for t in ctx.tune_read()],
                  "finite": bool(torch.isfinite(out).all()), "close": float((out.cpu() - ref).norm() / ref.norm())}))
"""


def test_timed_once_there_is_memory(tmp_path):
    env = dict(os.environ, PK_TUNE_FILE=str(tmp_path / "tune.txt"), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CODE], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout.strip().splitlines()[-1])
    assert d["tight"] == [0, 0]              # no decision while memory is short
    assert d["later"] >= 3 and set(d["sources"]) == {"timed"}
    assert d["finite"] and d["close"] < 1e-6

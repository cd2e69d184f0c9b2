"""The environment switches of the GEMM kernels, read once per process: each is looked at in one of its own. Plans need no GPU."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SIZES = [(256, 768, 256), (1000, 2568, 5160), (4096, 4096, 4096)]
PLANS = """
import ctypes, json
from aws_ofi_nccl_b200.ops import _lib
lib, ll, vp = _lib.load(), ctypes.c_longlong, ctypes.c_void_p
out = {"joint": [], "mlp": []}
for M, N, K in %r:
    r = [ctypes.c_int() for _ in range(3)]
    assert lib.b200_linear_grads_plan(M, N, K, *(ctypes.byref(x) for x in r)) == 0
    out["joint"].append(r[0].value)
    out["mlp"].append([lib.b200_gemm_swiglu_launches(vp(4096), vp(4096), M, N, K, ll(K)), lib.b200_gemm_swiglu_bwd_launches(vp(4096), vp(4096), M, N, K, ll(K))])
out["group"] = lib.b200_linear_grads_group(4096, 4096, 4096)
print(json.dumps(out))
""" % SIZES


def _plans(**env):
    e = {k: v for k, v in os.environ.items() if not k.startswith("B200_GEMM_")}
    r = subprocess.run([sys.executable, "-c", PLANS], capture_output=True, text=True, timeout=300, cwd=ROOT, env={**e, **env})
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout)


@pytest.mark.parametrize("env,joint,mlp", [({}, 1, [1, 1]), ({"B200_GEMM_2CTA": "0"}, 0, [2, 2])])
def test_without_pairs_no_product_runs_on_them(env, joint, mlp):
    plans = _plans(**env)
    assert plans["joint"] == [joint] * len(SIZES) and plans["mlp"] == [mlp] * len(SIZES)


@pytest.mark.parametrize("env,group", [({}, 8), ({"B200_GEMM_GROUP_M": "0"}, 0), ({"B200_GEMM_GROUP_M": "5"}, 3)])
def test_the_raster_group_of_joint_gradients(env, group):
    """In tiles of 256 rows, where the variable counts 128."""
    assert _plans(**env)["group"] == group

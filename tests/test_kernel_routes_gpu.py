"""Which kernels a call runs, by their names: the tests that compare two walks bit for bit would not notice if both were one.
The names come from the profiler in a process of its own (in a long one it loses records)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import json, os, sys
import torch
sys.path.insert(0, sys.argv[1])
from ojasx_b200 import ops, synth
mark = torch.zeros(1, device="cuda")

def names(call):
    call()
    for _ in range(8):
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            mark.erfinv_()
            call()
            mark.erfinv_()
            torch.cuda.synchronize()
        got = [e.name for e in p.events() if not e.name.startswith("cuda")]
        if sum("erfinv" in n for n in got) == 2:      # the record is whole
            return " ".join(got)
    return None

def run(name, call, **env):
    os.environ.update(env)
    out[name] = names(call)
    for k in env:
        del os.environ[k]

def randn(*shape):
    return torch.randn(*shape, generator=torch.Generator("cuda").manual_seed(1), device="cuda")

out = {"sms": torch.cuda.get_device_properties(0).multi_processor_count}
for K, M, batch, frac in ((4096, 2560, 128, 0.0), (4096, 2560, 256, 0.0), (1024, 4096, 32, 0.0), (1024, 4096, 512, 0.05)):
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(7, K, M, block_dim=8, outlier_frac=frac))
    x = randn(batch, K)
    run(f"linear {K} {M} {batch} {frac}", lambda: layer(x))
run("linear rows", lambda: layer(x), OJASX_B200_LINEAR_WALK="rows")
moe = ops.VQMoE(synth.make_vq_moe(1, 12, 2560, 640, block_dim=8, outlier_frac=0.0))
for tokens, k in ((1, 10), (4, 8), (8, 8)):
    x2 = randn(tokens, 2560)
    run(f"few {tokens * k}", lambda: moe.forward_routed(x2, k))
x3 = randn(32, 2560)
one = dict(OJASX_B200_MOE_QUAD_MIN_PAIRS=str(1 << 30))
run("chain", lambda: moe.forward_routed(x3, 10), **one)
run("chain two", lambda: moe.forward_routed(x3, 10), OJASX_B200_MOE_ONE_LAUNCH="0", **one)
run("rows", lambda: moe.forward_routed(x3, 10), OJASX_B200_MOE_CHAIN="0", **one)
run("quad", lambda: moe.forward_routed(x3, 10), OJASX_B200_MOE_QUAD_MIN_PAIRS="1")
print(json.dumps(out))
"""


def test_routes(cuda):
    run = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    ran = json.loads(run.stdout.strip().splitlines()[-1])
    sms = ran.pop("sms")
    if None in ran.values():
        pytest.skip("the profiler records no kernels")

    def has(name, *kernels):
        return [k in ran[name] for k in kernels]

    assert has("linear rows", "lut_linear_quad_kernel", "lut_linear_kernel") == [False, True]
    assert has("chain", "moe_experts_chain_kernel", "quad") == [True, False]
    assert has("chain two", "moe_gate_up_chain_kernel", "moe_down_chain_kernel", "moe_experts_chain_kernel") == [True, True, False]
    assert has("rows", "chain", "quad", "moe_gate_up_kernel") == [False, False, True]
    assert has("quad", "moe_gate_up_quad_kernel", "moe_down_quad_kernel") == [True, True]
    if sms != 148:
        return            # the estimates depend on it
    # us with one vector and with four: 80.3 / 92.8; 158 / 114; and the layer's own outliers count
    assert [has(f"linear {c}", "lut_linear_quad_kernel")[0] for c in ("4096 2560 128 0.0", "4096 2560 256 0.0", "1024 4096 32 0.0", "1024 4096 512 0.05")] \
        == [False, True, False, True]
    # us by the row-per-lane kernels and by those for a handful of pairs: 40.8 / 32.7, 71.4 / 70.2, 83.9 / 113.5
    few = ("moe_gate_up_few_kernel", "moe_down_few_kernel")
    assert [has(f"few {n}", *few) for n in (10, 32, 64)] == [[True, True], [True, True], [False, False]]

"""FSA_CHECK_STATUS=1 covers the layer's native function: every status word is read after its launches, and a non-zero one raises.
The failure is an error code from a stand-in for ``fsa_read_status`` that the host code finds before the library's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SHIM = r"""
int reads = 0, fail_at = -1;
int fsa_read_status(const void* word, void* stream, int* out) {
    if (!word) return -1;
    *out = reads == fail_at;
    return reads++ == fail_at ? -5 : 0;
}
"""

SCRIPT = r"""
import ctypes, os, sys
shim = ctypes.CDLL(sys.argv[1], mode=os.RTLD_GLOBAL | os.RTLD_NOW)
reads, fail_at = (ctypes.c_int.in_dll(shim, n) for n in ("reads", "fail_at"))
sys.path.insert(0, sys.argv[2])
import torch
from fsa.module.fsa import FlashSparseAttention, RopeConfig
layer = FlashSparseAttention(256, 4, 2, 128, 32, 16, 64, 6, 1, 2, 128, rope_config=RopeConfig(head_dim=128)).cuda().to(torch.bfloat16)
x = torch.randn(300, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
cu = torch.tensor([0, 300], dtype=torch.int32, device="cuda")
def step():
    layer(x, cu, [300]).float().sum().backward()
step()
n = reads.value
print("reads", n)
for i in range(n):
    reads.value, fail_at.value = 0, i
    try:
        step()
        print("silent", i)
    except RuntimeError as e:
        print("raised", str(e).split(" status")[0])
"""


def test_layer_reads_the_status_of_its_kernels(tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c")], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(tmp_path / "shim.so"), os.path.join(HERE, "..", "flash-sparse-attention_b200")],
                       env={**os.environ, "FSA_CHECK_STATUS": "1"}, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    said = r.stdout.split("\n")
    assert "silent" not in r.stdout
    assert sorted(x.removeprefix("raised ") for x in said if x.startswith("raised")) == [
        "fsa_compress_kv_bwd", "fsa_compress_kv_fwd", "fsa_range_attn_bwd_delta", "fsa_range_attn_bwd_delta", "fsa_sel_bwd_delta", "fsa_sel_fwd",
        "range attention and block selection"], r.stdout

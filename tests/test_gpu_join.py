"""A batch that goes in two halves on two streams, when the caller's stream cannot be made to wait for the second: the call
must report it, and must not return while the half runs on. The failing call is a fake: the library's objects are linked
once more with one function of the CUDA runtime wrapped, which returns an error code for one stream instead of calling on."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FAKE = r"""
static void* refused = 0;
static int count     = 0;
int __real_cudaStreamWaitEvent(void* stream, void* event, unsigned flags);
int __wrap_cudaStreamWaitEvent(void* stream, void* event, unsigned flags)
{
  if (refused != 0 && stream == refused) {
    count++;
    return 999;  /* cudaErrorUnknown */
  }
  return __real_cudaStreamWaitEvent(stream, event, flags);
}
__attribute__((visibility("default"))) int refuse_waits(void* stream)
{
  const int before = count;
  refused          = stream;
  count            = 0;
  return before;
}
"""

CHILD = r"""
import ctypes as C
import sys
import numpy as np
import torch
sys.path[:0] = [ROOT, ROOT + "/tests"]
from octex_b200 import _lib, synth
from test_gpu_paths import make_index, same, search_at
dim, k, n = 64, 10, 2800
idx, _ = make_index(dim, copies=6, blocks=4)
kw = dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)
queries = torch.as_tensor(synth.plumbing(n, dim, seed=6), device="cuda")
want = [t.cpu().numpy() for t in idx.search(queries, k, **kw)]
ids, dist = torch.empty((n, k), dtype=torch.int64, device="cuda"), torch.empty((n, k), device="cuda")
side = torch.cuda.Stream()
refuse = _lib.lib().refuse_waits
refuse.argtypes = [C.c_void_p]


def call():
    ids.fill_(-5)
    torch.cuda.synchronize()
    search_at(idx, queries.data_ptr(), ids.data_ptr(), dist.data_ptr(), n, dim, k, wait=False, stream=side.cuda_stream, **kw)


call()  # the plan's batch before is on the same stream: the call waits for nothing but its half
side.synchronize()
assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
refuse(side.cuda_stream)
failed = False
try:
    call()
except RuntimeError as e:
    failed = "CUDA error" in str(e)
refused = refuse(None)
assert refused > 0, "no wait was refused: the batch did not go in halves"
assert failed, "a call whose halves were not joined returned without an error"
side.synchronize()  # not the stream of the second half
assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
call()
side.synchronize()
assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
idx.close()
print("joined")
"""


def test_halves_that_cannot_be_joined(tmp_path):
    from octex_b200 import _build
    _build.build()
    objects = [os.path.join(_build.LIB_DIR, s.replace(".cu", ".o")) for s in _build.SOURCES]
    (tmp_path / "fake.c").write_text(FAKE)
    fake, lib = str(tmp_path / "fake.o"), str(tmp_path / "with_fake.so")
    subprocess.check_call(["gcc", "-O1", "-fPIC", "-c", str(tmp_path / "fake.c"), "-o", fake])
    subprocess.check_call([_build._nvcc(), "-shared", "-o", lib] + objects + [fake, "-Xlinker", "--wrap=cudaStreamWaitEvent",
                                                                              "-lcudart_static", "-lpthread", "-ldl", "-lrt"])
    child = subprocess.run([sys.executable, "-c", CHILD.replace("ROOT", repr(_build._ROOT))], capture_output=True, text=True,
                           timeout=300, env=dict(os.environ, OCTEX_B200_LIB=lib))
    assert child.returncode == 0 and child.stdout.strip() == "joined", child.stderr[-2000:]

"""Other Python threads run while the host extension is inside an entry point. The extension is loaded beside a stand-in for the
kernel library whose convolution waits half a second, so the test needs no GPU."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from maxdiffusion_b200 import build

_STUB = r"""
#include <c10/cuda/CUDAStream.h>
#include <unistd.h>
namespace c10::cuda {
CUDAStream getCurrentCUDAStream(DeviceIndex) { return CUDAStream(CUDAStream::UNCHECKED, Stream(Stream::DEFAULT, Device(kCUDA, 0))); }
cudaStream_t CUDAStream::stream() const { return nullptr; }
}
extern "C" {
int mdb_conv_igemm(...) { usleep(500000); return 0; }
#define NOT_CALLED(name) int name(...) { return 9999; }
NOT_CALLED(mdb_flash_fwd) NOT_CALLED(mdb_flash_fwd_d64) NOT_CALLED(mdb_flash_fwd_narrow) NOT_CALLED(mdb_geglu_fwd)
NOT_CALLED(mdb_gemm_bf16) NOT_CALLED(mdb_gemm_geglu) NOT_CALLED(mdb_gemm_group) NOT_CALLED(mdb_gn_cl_apply)
NOT_CALLED(mdb_gn_cl_fold_fwd) NOT_CALLED(mdb_gn_cl_sums) NOT_CALLED(mdb_ln_fwd) NOT_CALLED(mdb_rms_rope_fwd)
}
"""

_RUN = r"""
import ctypes, importlib.util, sys, threading, time
import torch
spec = importlib.util.spec_from_file_location("_host_ops", sys.argv[1])
host = importlib.util.module_from_spec(spec)
spec.loader.exec_module(host)
host.setup(RuntimeError, lambda *a: (1, 64, 1))
ticks, stop = [], threading.Event()
def tick():
  while not stop.is_set():
    ticks.append(time.monotonic())
    time.sleep(0.005)
thread = threading.Thread(target=tick)
thread.start()
time.sleep(0.1)
table = (ctypes.c_int * 8)()
x = torch.zeros(4)
begin = time.monotonic()
out = host.conv(x, None, torch.zeros(2, 2), x, None, None, (1,) * 5, (1,) * 4, (1,) * 5, (1,) * 4, (1,) * 3, (1,) * 4, 8, 8,
                ctypes.addressof(table), ctypes.addressof(table), -1, 0, (1,) * 4, (0,), 0, 1, 64, 1, 1, 1)
end = time.monotonic()
stop.set()
thread.join()
assert out is x and end - begin > 0.4 and host.launches() == 1
print(sum(begin + 0.05 < t < end - 0.05 for t in ticks))
"""


def test_other_threads_run_during_a_launch(tmp_path):
  cuda = Path("/usr/local/cuda")
  if not build.HOST_PATH.exists() or shutil.which("g++") is None or not (cuda / "include" / "cuda_runtime_api.h").exists():
    pytest.skip("the host extension is not built, or there is nothing to build the stand-in with")
  root = Path(torch.__file__).resolve().parent
  (tmp_path / "stub.cpp").write_text(_STUB)
  res = subprocess.run(["g++", "-std=c++17", "-O0", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                        "-I", str(root / "include"), "-I", str(root / "include" / "torch" / "csrc" / "api" / "include"), "-I",
                        str(cuda / "include"), str(tmp_path / "stub.cpp"), "-o", str(tmp_path / "_kernels.so")], capture_output=True, text=True)
  assert res.returncode == 0, res.stderr
  shutil.copy(build.HOST_PATH, tmp_path / "_host_ops.so")
  env = {k: v for k, v in os.environ.items() if k != "LD_LIBRARY_PATH"}
  res = subprocess.run([sys.executable, "-c", _RUN, str(tmp_path / "_host_ops.so")], capture_output=True, text=True, env=env, timeout=300)
  assert res.returncode == 0, res.stderr
  assert int(res.stdout) > 20  # 80 ticks of 5 ms fit into the half second

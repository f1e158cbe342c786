"""The CTAs of a cluster leave the kernel together: when some of them fail, the
others find out at the next barrier they pass, not earlier and not later, and
all are gone after it.  The failures are decided by the host (a list of ranks
and the step at which each gives up); every loop is bounded.  The device
functions are compiled from the library's own sources with its own flags."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from coldplate_solver_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "cps_device.cuh"
// As in the batch kernel: each step is a reduction; out[rank]: barriers passed by a CTA that left, -1 if it ran to the end.
__global__ void __launch_bounds__(cps::kThreads) by_barrier(const int* when, int steps, int* out) {
  __shared__ double smem[cps::kRedWidth * 8], redbuf[2 * cps::kRedWidth];
  cps::cg::cluster_group cl = cps::cg::this_cluster();
  cps::ClusterGroup g{redbuf, nullptr, cl.block_rank(), cl.num_blocks(), 0u, 0u, false};
  if (threadIdx.x == 0) cps::s_cluster_leave = cps::kStay;
  g.sync();
  int left = -1;
  for (int k = 0; k < steps && left < 0; ++k) {
    if (when[g.rank] == k) {
      cps::cluster_leave(true, g.barriers + 1);
      left = (int)g.barriers + 1;
      break;
    }
    double v[1] = {1.0};
    if (!g.sync_reduce<1, 0u>(v, smem)) left = (int)g.barriers;
    else if (v[0] != (double)g.nblk * cps::kThreads) left = 1000;
  }
  if (left < 0) cl.sync();
  if (threadIdx.x == 0) out[g.rank] = left;
}
// As in the grid form: a step may fail before the two barriers of its inner loop's pass, whose first one tells.
__global__ void __launch_bounds__(cps::kThreads) by_word(const int* when, int steps, int* out) {
  const unsigned rank = cps::cg::this_cluster().block_rank();
  cps::cluster_enter();
  int left = -1;
  for (int k = 0; k < steps && left < 0; ++k) {
    if (when[rank] == k) {
      cps::cluster_leave(true);
      left = k;
      break;
    }
    cps::cluster_arrive();
    cps::cluster_wait();
    if (cps::cluster_leaving()) {
      left = k;
      break;
    }
    cps::cluster_arrive();
    cps::cluster_wait();
  }
  if (left < 0) cps::cluster_leave(false);
  if (threadIdx.x == 0) out[rank] = left;
}
extern "C" int run(int word, int ctas, const int* when, int steps, int* out) {
  const void* fn = word ? (const void*)by_word : (const void*)by_barrier;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(cps::kThreads);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&when, &steps, &out};
  if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, fn, args);
  return (int)(e == cudaSuccess ? cudaDeviceSynchronize() : e);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("cluster_leave")
    src, so = tmp / "leave.cu", tmp / "leave.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", os.path.join(build.PKG_DIR, "csrc"), "-o", str(so), str(src)],
                   check=True)
    h = ctypes.CDLL(str(so))
    p = ctypes.c_void_p
    h.run.argtypes = [ctypes.c_int, ctypes.c_int, p, ctypes.c_int, p]
    return h


@pytest.mark.parametrize("word", [0, 1])
@pytest.mark.parametrize("ctas", [1, 2, 8, 16])
@pytest.mark.parametrize("failing", [(), (0,), (-1,), (0, -1), "all"])
def test_a_cluster_leaves_together(lib, word, ctas, failing):
    import torch
    steps, at = 40, 17
    ranks = range(ctas) if failing == "all" else sorted({r % ctas for r in failing})
    when = np.full(ctas, -1, np.int32)
    for r in ranks:
        when[r] = at
    dev = torch.from_numpy(when).cuda()
    out = torch.full((ctas,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(20):
        assert lib.run(word, ctas, dev.data_ptr(), steps, out.data_ptr()) == 0
        got = out.cpu().numpy()
        # the barrier before the first step, one per step before, and the one all leave at
        want = -1 if not len(ranks) else at if word else at + 2
        assert (got == want).all(), got

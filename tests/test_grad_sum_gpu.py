"""The gradient sum, Adam step and average where a CTA's row of sums never came (its
MMA wait ran out): the sum kernel alone, on rows made by hand."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from ssmdlbm_b200 import build

pytestmark = pytest.mark.gpu

_SUM = """
#include "adam.cuh"
constexpr int P = 70;
extern "C" int run(const float *rows, int ctas, long long n, float *grad, double *loss, float *net, float *m, float *v, float *avg) {
    ssmd::AdamArgs ad{net, m, v, avg, 1e-3f, 0.9f, 0.999f, 1e-8f, 0.1f, 0.001f, 0.9f};
    ssmd::grad_sum_kernel<P><<<(P + 1 + 31) / 32, ssmd::kSumThreads>>>(rows, ctas, n, grad, loss, ad);
    return (int)cudaDeviceSynchronize();
}
extern "C" unsigned mark() { return ssmd::kAbortedRow; }
"""


def test_a_row_that_never_came_changes_no_weights(tmp_path):
    if not (os.environ.get("NVCC") or shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")):
        pytest.skip("needs nvcc")
    src, so = tmp_path / "sum.cu", tmp_path / "sum.so"
    src.write_text(_SUM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-shared", "-Xcompiler", "-fPIC", "-cudart", "static",
                    "-o", str(so), str(src)], check=True, capture_output=True)
    run = ctypes.CDLL(str(so))
    run.run.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong] + [ctypes.c_void_p] * 6
    P = 70
    for ctas in (1, 33, 256):
        for at in (None, 0, ctas - 1):
            rows = np.random.default_rng(ctas).normal(0, 1, (ctas, P + 1)).astype(np.float32)
            want = np.zeros(P, np.float32)
            for r in rows:
                want += r[:P]  # FP32, in CTA order
            if at is not None:
                rows.view(np.uint32)[at, P] = run.mark()
            dr = torch.as_tensor(rows, device="cuda")
            start = {k: torch.rand(P, device="cuda") for k in ("net", "m", "v", "avg")}
            t = {k: v.clone() for k, v in start.items()}
            grad, loss = torch.zeros(P, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert run.run(dr.data_ptr(), ctas, 10, grad.data_ptr(), loss.data_ptr(), *(t[k].data_ptr() for k in ("net", "m", "v", "avg"))) == 0
            if at is None:
                assert np.array_equal(grad.cpu().numpy(), want)
                assert abs(loss.item() - rows[:, P].astype(np.float64).sum() / 10) <= 1e-12 * np.abs(rows[:, P]).sum()
                assert all((t[k] != start[k]).any() for k in t)
            else:
                assert grad.isnan().all() and loss.isnan().all()
                assert all(torch.equal(t[k], start[k]) for k in t)

"""torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False reaches the matrix products that the
native mixer and stack hand to cuBLAS directly (GPU). The library's results need not show it, so a preloaded
cublasGemmEx looks at the handle's math mode at every call."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SHIM = r"""
#define _GNU_SOURCE
#include <cublas_v2.h>
#include <dlfcn.h>
static int calls, strict;
int seen_calls(void) { return calls; }
int seen_strict(void) { return strict; }
static void* library(const char* name) { return dlsym(dlopen("libcublas.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
cublasStatus_t cublasGemmEx(cublasHandle_t h, cublasOperation_t ta, cublasOperation_t tb, int m, int n, int k,
                            const void* alpha, const void* a, cudaDataType at, int lda, const void* b, cudaDataType bt,
                            int ldb, const void* beta, void* c, cudaDataType ct, int ldc, cublasComputeType_t compute,
                            cublasGemmAlgo_t algo) {
    cublasMath_t mode = CUBLAS_DEFAULT_MATH;
    ((cublasStatus_t (*)(cublasHandle_t, cublasMath_t*))library("cublasGetMathMode"))(h, &mode);
    ++calls;
    if (mode & CUBLAS_MATH_DISALLOW_REDUCED_PRECISION_REDUCTION) ++strict;
    cublasStatus_t (*next)() = (cublasStatus_t (*)())library("cublasGemmEx");
    return next(h, ta, tb, m, n, k, alpha, a, at, lda, b, bt, ldb, beta, c, ct, ldc, compute, algo);
}
"""

CHILD = r"""
import ctypes, sys, torch
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import mirror
from fields_lm_b200 import mixer
shim = ctypes.CDLL({shim!r})
m = mirror.IndependentVacancyField(256).cuda()
x = torch.randn(2, 33, 256, device="cuda", requires_grad=True)
for allowed in (True, False):
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = allowed
    calls, strict = shim.seen_calls(), shim.seen_strict()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = mixer.fused_mixer_forward(m, x)
    y.sum().backward()
    torch.cuda.synchronize()
    calls, strict = shim.seen_calls() - calls, shim.seen_strict() - strict
    assert calls > 0 and strict == (0 if allowed else calls), (allowed, calls, strict)
print("seen")
"""


def test_products_heed_the_reduction_setting(tmp_path):
    source, shim = tmp_path / "shim.c", tmp_path / "libshim.so"
    source.write_text(SHIM)
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", f"-I{home}/include", "-o", str(shim), str(source), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(shim))
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT), shim=str(shim))], env=env,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "seen" in out.stdout, out.stdout + out.stderr

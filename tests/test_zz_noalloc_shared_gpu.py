"""The allocation-free join beside another kernel that holds most of the GPU:
it runs in the room that is left and does not wait for the other to end."""
import ctypes
import subprocess
import time

import numpy as np
import pytest

SRC = r"""
#include <stdint.h>
// Holds the CTA's threads for `us` microseconds (and 4M naps at most).
__global__ void __launch_bounds__(1024) hold(uint64_t us) {
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t i = 0; i < 4000000u; i++) {
        __nanosleep(2000);
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > us * 1000) break;
    }
}
extern "C" int hold_on(int ctas, uint64_t us, void* stream) {
    hold<<<ctas, 1024, 0, (cudaStream_t)stream>>>(us);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import build
    d = tmp_path_factory.mktemp("hold")
    src, so = str(d / "hold.cu"), str(d / "hold.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build._nvcc()] + build.NVCC_FLAGS + ["-shared", src, "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.hold_on.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p]
    return L


@pytest.mark.gpu
def test_noalloc_runs_beside_a_long_kernel(built, lib):
    import torch

    import dim3gpu
    from oracle import oracle_py as O
    rng = np.random.default_rng(11)
    R, S = (rng.integers(0, 60_000, (n, 2)).astype(np.uint32) for n in (150_000, 90_000))
    want, n, _, _ = O.join_project(R, S)
    dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    L, vp, u64 = dim3gpu.load(), ctypes.c_void_p, ctypes.c_uint64
    L.dim3g_join_project_noalloc.argtypes = [vp, u64, vp, u64, vp, u64, ctypes.POINTER(u64), vp]
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()

    def join():
        got = u64()
        rc = L.dim3g_join_project_noalloc(dR.data_ptr(), R.shape[0], dS.data_ptr(), S.shape[0], out.data_ptr(), n,
                                          ctypes.byref(got), mine.cuda_stream)
        assert rc == dim3gpu.OK and got.value == n

    torch.cuda.synchronize()
    join()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    done = torch.cuda.Event()
    hold_ms = 400
    t = time.perf_counter()
    assert lib.hold_on(2 * (sms - 12), hold_ms * 1000, other.cuda_stream) == 0  # 1024 threads a CTA, two an SM
    done.record(other)
    time.sleep(0.02)
    join()
    ms = 1e3 * (time.perf_counter() - t)
    assert not done.query() and ms < hold_ms / 2, ms
    torch.cuda.synchronize()
    assert np.array_equal(np.sort(O.pair_keys(out.cpu().numpy().view(np.uint32))), np.sort(O.pair_keys(want)))

"""CPU: the integer rounding of FP64 to FP32 against the conversion, bit for bit."""
import ctypes
import os
import subprocess

import numpy as np

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "state_estimation_with_cuda_gb300",
                      "csrc", "kernels")
SRC = r'''
#include "round32.h"
extern "C" void run(const uint64_t* v, long n, uint32_t* out, unsigned char* takes) {
    for (long i = 0; i < n; ++i) {
        const uint32_t hi = static_cast<uint32_t>(v[i] >> 32), lo = static_cast<uint32_t>(v[i]);
        takes[i] = sle_gb300::round32_takes(hi);
        out[i] = sle_gb300::round32_bits(hi, lo);
    }
}
'''


def test_round32_equals_the_conversion(tmp_path):
    (tmp_path / "r.cpp").write_text(SRC)
    so = tmp_path / "r.so"
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I", HEADER, str(tmp_path / "r.cpp"), "-o", str(so)])
    rng = np.random.default_rng(5)
    exp = np.concatenate([np.repeat(np.arange(890, 900), 4096), np.repeat(np.arange(1144, 1156), 4096),
                          rng.integers(0, 2048, 100000)]).astype(np.uint64)
    man = rng.integers(0, 1 << 52, exp.size, dtype=np.uint64)
    kind = rng.integers(0, 5, exp.size)  # any; a tie; one off a tie either way; all ones above the cut
    tie = (man & ~np.uint64((1 << 29) - 1)) | np.uint64(1 << 28)
    man = np.select([kind == 1, kind == 2, kind == 3, kind == 4],
                    [tie, tie + np.uint64(1), tie - np.uint64(1), man | np.uint64(((1 << 23) - 1) << 29)], man)
    bits = (rng.integers(0, 2, exp.size, dtype=np.uint64) << np.uint64(63)) | (exp << np.uint64(52)) | man
    bits = np.concatenate([bits, np.array([0, 1 << 63, 0x7FF0 << 48, 0x7FF8 << 48, 1], dtype=np.uint64)])
    out = np.empty(bits.size, np.uint32)
    takes = np.empty(bits.size, np.uint8)
    ctypes.CDLL(str(so)).run(bits.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(bits.size),
                             out.ctypes.data_as(ctypes.c_void_p), takes.ctypes.data_as(ctypes.c_void_p))
    with np.errstate(over="ignore", invalid="ignore"):
        ref = bits.view(np.float64).astype(np.float32)
    e = (bits >> np.uint64(52)) & np.uint64(0x7FF)
    assert np.array_equal(takes != 0, (e >= 897) & (e <= 1150))
    assert (takes != 0).sum() > 20000
    assert np.array_equal(out[takes != 0], ref.view(np.uint32)[takes != 0])

"""The six digit rows of a quantised value (csrc/s14_umma.cuh, digit6_code_bytes): the function's source, built for the host, over every
E4M3FN value at every exponent that its scale block can have."""
import ctypes as C
import os
import re
import shutil
import subprocess

from colormlm_b200 import build

E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]
SHIM = r"""
#include <cstdint>
// the byte permutation of the PTX instruction: nibble i of sel picks byte (nibble & 7) of {a, b}
static uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    const uint64_t ab = (uint64_t)b << 32 | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) {
        const uint32_t n = sel >> (4 * i) & 15u, byte = (uint32_t)(ab >> (8 * (n & 7u))) & 255u;
        r |= (n & 8u ? (byte & 128u ? 255u : 0u) : byte) << (8 * i);
    }
    return r;
}
#define __device__
#define __forceinline__ inline
"""


def test_every_value_at_every_exponent(tmp_path):
    source = open(os.path.join(build.CSRC, "s14_umma.cuh")).read()
    function = re.search(r"__device__ __forceinline__ void digit6_code_bytes\(.*?\n}\n", source, re.S).group(0)
    (tmp_path / "d.cpp").write_text(SHIM + function + 'extern "C" void digits(int q, uint32_t *c) { digit6_code_bytes(q, c[0], c[1]); }\n')
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(tmp_path / "d.so"), str(tmp_path / "d.cpp")],
                   check=True)
    lib, out, cases = C.CDLL(str(tmp_path / "d.so")), (C.c_uint32 * 2)(), 0
    for code in range(127):                          # (the 128th is the NaN)
        mantissa, exponent = code & 7, code >> 3
        steps = mantissa if exponent == 0 else (8 + mantissa) << (exponent - 1)   # the value as a multiple of 2^-9
        least = max(steps.bit_length() - 9, -8) if steps else -8                  # |v| < 2^E
        for E in range(least, 10):                   # 448 < 2^9: no block of E4M3FN values has a larger exponent
            q, rest = divmod(steps << (18 + 9), 1 << (9 + 9 + E))                 # v 2^(18 - E)
            assert rest == 0
            for sign in (1, -1):
                lib.digits(C.c_int(sign * q), out)
                codes = [out[0] >> (8 * j) & 255 for j in range(4)] + [out[1] & 255, out[1] >> 8 & 255]
                assert all(c < 16 for c in codes) and out[1] < 1 << 16
                values = [(-1.0 if c & 8 else 1.0) * E2M1[c & 7] for c in codes]
                assert 2.0 * sum(v * 8.0 ** j for j, v in enumerate(values)) == sign * q, (code, E, sign, codes)
                cases += 1
    assert cases > 2000

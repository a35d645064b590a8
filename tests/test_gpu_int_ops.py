"""The FP64 form's products, quotients and roots on the integer pipes, and its quotients by a
prepared reciprocal, operand by operand against the FP64 unit: equal bits (no tolerance), over
random significands, short ones (exact results and ties), ones next to powers of two, and
quotients and roots next to a midpoint between two results."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SRC = r"""
#include "tsg_pairs64.cuh"
using namespace tsg;
// which of the four a pair fails in, and how many were compared
__global__ void k_check(const double* a, const double* b, int n, unsigned long long* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const auto differ = [](double x, double y) { return __double_as_longlong(x) != __double_as_longlong(y); };
    const double x = a[i], y = b[i], v = fabs(x), w = fabs(y);
    if (usable(x) && usable(y)) {
        atomicAdd(&out[4], 1ull);
        if (differ(int_mul(x, y), x * y)) atomicAdd(&out[0], 1ull);
    }
    const unsigned long long X = divisor(w);
    if (X != 0ull && usable(x) && !zero(x)) {
        atomicAdd(&out[5], 1ull);
        if (differ(int_quot(x, w, X), x / w)) atomicAdd(&out[1], 1ull);
    }
    if (usable(v) && !zero(v)) {
        atomicAdd(&out[6], 1ull);
        if (differ(int_sqrt(v), sqrt(v))) atomicAdd(&out[2], 1ull);
    }
    if (w > 0x1p-200 && w < 0x1p200) {
        atomicAdd(&out[7], 1ull);
        if (differ(div_by(x, w, __drcp_rn(w), 1000u << 20), x / w)) atomicAdd(&out[3], 1ull);
    }
}
extern "C" int check(const double* a, const double* b, int n, unsigned long long* out) {
    k_check<<<(n + 255) / 256, 256>>>(a, b, n, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def check(native, tmp_path_factory):
    from tisphi_gb300 import build_native as bn
    d = tmp_path_factory.mktemp("int_ops")
    src, lib = d / "int_ops.cu", d / "libint_ops.so"
    src.write_text(SRC)
    subprocess.run([bn._nvcc(), *bn.ARCH, "-O3", "-std=c++17", "-fmad=false", "--extended-lambda", "-I", bn.CSRC, "-I",
                    bn.INCLUDE, "-shared", "-Xcompiler", "-fPIC", str(src), "-o", str(lib), "-lcudart"], check=True)
    fn = ctypes.CDLL(str(lib)).check
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    return fn


def _significands(kind, rng, n):
    """53-bit integers in [2^52, 2^53)."""
    full = rng.integers(1 << 52, 1 << 53, n)
    if kind == "random":
        return full
    if kind == "short":  # few leading bits: exact products and ties
        return full & ~((np.int64(1) << rng.integers(20, 53, n)) - 1)
    edge = rng.integers(0, 8, n)  # next to a power of two
    return np.where(rng.random(n) < 0.5, (1 << 52) + edge, (1 << 53) - 1 - edge)


def _double(m, e, rng):
    x = np.ldexp(m.astype(np.float64), e - 52)
    return np.where(rng.random(m.size) < 0.5, -x, x)


N = 1 << 20


def _operands(kind, spread, rng):
    """|exponents| up to `spread`; 300 leaves the usable range on both sides."""
    if kind in ("midpoint_quotient", "midpoint_root"):
        # x next to (k + 1/2) w, or to (k + 1/2)^2: built in exact integers
        k = rng.integers(1 << 52, 1 << 53, N)
        w = rng.integers(1 << 52, 1 << 53, N)
        if kind == "midpoint_root":
            sq = [(2 * int(q) + 1) ** 2 for q in k[: 1 << 16]]  # 107 or 108 bits
            xs = np.array([float(s >> (s.bit_length() - 53)) for s in sq])
            a = np.ldexp(np.tile(xs, N >> 16), rng.integers(-spread, spread + 1, N) - 52)
            a = np.nextafter(a, np.where(rng.random(N) < 0.5, np.inf, 0.0))
            return a, _double(w, rng.integers(-spread, spread + 1, N), rng)
        pr = [(2 * int(q) + 1) * int(v) for q, v in zip(k[: 1 << 16], w[: 1 << 16])]
        xs = np.tile(np.array([float(s >> (s.bit_length() - 53)) for s in pr]), N >> 16)
        e = rng.integers(-spread, spread + 1, N)
        b = np.ldexp(np.tile(w[: 1 << 16].astype(np.float64), N >> 16), -52)
        return np.ldexp(xs, e - 52) * np.where(rng.random(N) < 0.5, -1.0, 1.0), b
    a = _double(_significands(kind, rng, N), rng.integers(-spread, spread + 1, N), rng)
    b = _double(_significands(kind, rng, N), rng.integers(-spread, spread + 1, N), rng)
    a[:: 1009] = 0.0
    b[:: 997] = -0.0
    return a, b


@pytest.mark.parametrize("kind", ["random", "short", "edge", "midpoint_quotient", "midpoint_root"])
@pytest.mark.parametrize("spread", [2, 190, 300])
def test_equal_bits(check, kind, spread):
    rng = np.random.default_rng([spread, len(kind)])
    a, b = _operands(kind, spread, rng)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.zeros(8, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert check(ta.data_ptr(), tb.data_ptr(), N, out.data_ptr()) == 0
    out = out.tolist()
    assert out[:4] == [0] * 4, f"products, quotients, roots, prepared quotients that differ: {out}"
    assert min(out[4:]) > N // 4, out

"""The exponentials of attention: the polynomial is as close as ``ex2.approx``, and neither bf16 kernels nor e4m3 kernels set to ``ex2.approx``
lose a score that is not finite."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import codec, ops
from tests import util
from tests.test_gpu_kernels import T, f32, qb  # noqa: F401

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "quark_b200" / "csrc"
# a thread takes a pair of x[0 .. n): both functions of attn_common.cuh on the same values
HARNESS = """
#include "attn_common.cuh"
__global__ void pairs(const float* x, float* poly, float* approx, int n) {
  const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i + 1 >= n) return;
  float a = x[i], b = x[i + 1];
  qb::ex2_poly_f32x2(a, b);
  poly[i] = a;
  poly[i + 1] = b;
  approx[i] = qb::ex2_approx(x[i]);
  approx[i + 1] = qb::ex2_approx(x[i + 1]);
}
extern "C" int run(const float* x, float* poly, float* approx, int n) {
  pairs<<<(n / 2 + 255) / 256, 256>>>(x, poly, approx, n);
  return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def exponentials(qb, tmp_path_factory):  # noqa: F811
    """x (f32) -> the polynomial's and ex2.approx's 2^x, by the kernels' own source."""
    tmp = tmp_path_factory.mktemp("exponentials")
    (tmp / "pairs.cu").write_text(HARNESS)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", str(CSRC), "-shared", "-Xcompiler", "-fPIC", str(tmp / "pairs.cu"),
                    "-o", str(tmp / "pairs.so")], check=True, timeout=600)  # fmt: skip
    lib = ctypes.CDLL(str(tmp / "pairs.so"))
    lib.run.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]

    def run(x):
        assert x.size % 2 == 0
        xd, poly, approx = T(qb, x, "f32"), qb.QuarkTensor.empty(x.size, dtype="f32"), qb.QuarkTensor.empty(x.size, dtype="f32")
        qb.runtime.synchronize()
        assert lib.run(xd.data_ptr(), poly.data_ptr(), approx.data_ptr(), x.size) == 0
        return poly.to_numpy(), approx.to_numpy()

    return run


def test_the_polynomial_is_as_close_as_ex2_approx(exponentials):
    """Against 64 bits, within the 2^-22 that ex2.approx.f32 is documented to keep, over what scores are narrowed from: up to 2^8, and down to
    where the result is no longer a normal number."""
    x = np.concatenate([np.linspace(-125, 8, 1 << 18, dtype=np.float32), np.linspace(-2, 2, 1 << 16, dtype=np.float32), np.arange(-125, 9, 0.5, dtype=np.float32)])
    poly, _ = exponentials(x)
    want = np.exp2(x.astype(np.float64))
    assert np.abs(poly / want - 1).max() <= 2.0**-22
    np.testing.assert_array_equal(poly[x == np.rint(x)], want[x == np.rint(x)])  # the key that the maximum came from counts exactly 1


def test_the_polynomial_keeps_nan_and_underflow(exponentials):
    """What ex2.approx.ftz makes of NaN, of -inf and of what is too small for a normal number, in either place of a pair."""
    x = np.array([np.nan, -np.inf, -1e30, -127.4, -126.75, -126.5, -126.25, -126.01], np.float32)
    for at in (0, 1):
        pairs = np.zeros((x.size, 2), np.float32)
        pairs[:, at] = x
        poly, approx = exponentials(pairs.ravel())
        np.testing.assert_array_equal(poly, approx)
        assert np.isnan(poly[at]) and (poly.reshape(-1, 2)[1:, at] == 0).all() and (poly.reshape(-1, 2)[:, 1 - at] == 1).all()


# a cluster of key splits, one CTA per item, splits through the workspace, helpers
FORMS = [(12, 12, 8, 2, 11, 0), (12, 12, 8, 2, 11, 1), (12, 12, 8, 2, 11, 16), (8, 8, 16, 5, 240, 0)]


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("H,W,Hk,gqa,nb,splits", FORMS)
def test_a_key_that_is_not_finite_is_seen_at_every_position(qb, kv_dt, H, W, Hk, gqa, nb, splits):  # noqa: F811
    """A KV head holds one bad value in a key at position h of eight, somewhere or among the last keys (where tiles are masked).  NaN: all of the
    head's outputs are NaN.  Infinity (bf16): NaN where the score is +inf, and where it is -inf the bits that any score far below gives.  The
    other heads' bits do not change."""
    r = util.rng([77, H, nb])
    tpf, Hq, cap, ft = H * W, Hk * gqa, (nb + 1) * H * W, 1000
    make = util.bf16_randn if kv_dt == "bf16" else util.e4m3_randn
    qkv = util.bf16_randn(r, (tpf, (Hq + 2 * Hk) * 64))
    Kc, Vc = make(r, (Hk * cap, 64)), make(r, (Hk * 64, cap))
    segs, n = ops.compute_segments(ft, nb, tpf, 1)
    keys = np.concatenate([np.arange(segs[2 * i], segs[2 * i] + segs[2 * i + 1]) for i in range(n)])
    channel = 5
    anywhere = [h * cap + int(r.choice(keys[keys % 8 == h % 8])) for h in range(Hk)]
    at_the_end = [h * cap + int(keys[-8 + h % 8]) for h in range(Hk)]

    def run(K):
        return qb.qf.owl_attn(T(qb, qkv, "bf16"), T(qb, K, kv_dt), T(qb, Vc, kv_dt), T(qb, np.asarray(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, Hk, gqa, H, W,
                              nb, 1, compute_dtype=kv_dt, packed_qkv=True, frame_t=T(qb, np.array([ft], np.int32)), kv_splits=splits).to_numpy().reshape(tpf, Hk, gqa * 64)  # fmt: skip

    def planted(value, rows, which):
        K = Kc.copy()
        for h in which:
            K[rows[h], channel] = value
        return run(K)

    was = qb._lib.set_attn_exact_exp(True)
    try:
        clean = run(Kc)
        for rows, which in ((anywhere, range(Hk)), (at_the_end, range(Hk)), (anywhere, range(0, Hk, 3))):
            got = planted(0x7FC0 if kv_dt == "bf16" else 0x7F, rows, which)
            for h in range(Hk):
                if h in which:
                    assert np.isnan(f32(got[:, h], "bf16")).all(), h
                else:
                    np.testing.assert_array_equal(got[:, h], clean[:, h])
        if kv_dt == "e4m3":
            return
        q = f32(qkv[:, : Hq * 64], "bf16").reshape(tpf, Hq, 64).transpose(1, 0, 2)
        cos, sin = ops.rope_tables(H, W, ft, 64)
        y = ops.apply_rope(q, cos[None], sin[None])[..., channel].T.reshape(tpf, Hk, gqa)  # the sign of the score
        low, high = y < -0.05, y > 0.01
        assert low.any() and high.any()
        for rows in (anywhere, at_the_end):
            got = planted(0x7F80, rows, range(Hk)).reshape(tpf, Hk, gqa, 64)
            far = planted(int(codec.f32_to_bf16(np.array([1e6], np.float32))[0]), rows, range(Hk)).reshape(got.shape)
            assert np.isnan(f32(got, "bf16"))[high].all() and np.isfinite(f32(got, "bf16"))[low].all()
            np.testing.assert_array_equal(got[low], far[low])
    finally:
        qb._lib.set_attn_exact_exp(was)

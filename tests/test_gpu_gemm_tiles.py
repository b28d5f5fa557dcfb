"""The tile forms that ``qf.gemm`` chooses by size: pairs of CTAs for large products (with and without K slices), K slices summed
inside a cluster, and boxes of fewer than 128 rows; at sizes that leave remainders in rows, columns and K."""

import numpy as np
import pytest

from tests.test_gpu_kernels import _check_gemm, _gemm_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qb():
    import quark_b200 as q

    q._lib.require_device(0)
    yield q
    q.runtime.synchronize()
    assert q._lib.device_status() == 0


@pytest.mark.parametrize("M,N,K,fp8,kw", [
    # pairs, 128 and 256 columns: a last pair of which one CTA has no rows, column remainders, gate rows that change inside a tile
    (2300, 2120, 2048, True, dict(gate_groups=4)),
    (2300, 2120, 2048, False, dict(gate_groups=1)),
    (1700, 1800, 1600, False, dict(bias=True, act="silu", out_dtype="f32")),
    (2561, 3080, 1040, True, dict(out_dtype="e4m3", act="silu")),
    # pairs with K slices
    (300, 2048, 8192, False, dict(gate_groups=1)),
    (512, 2040, 8208, False, dict(gate_groups=2)),
    # K slices of a cluster over few rows
    (1, 2048, 2048, False, dict()),
    (13, 128, 4096, True, dict(bias=True)),
    (37, 520, 8192, True, dict(out_dtype="f32")),
    (128, 2048, 4096, True, dict(gate_groups=2)),
    (100, 136, 2064, False, dict(act="silu")),
])  # fmt: skip
def test_gemm_tile_forms(qb, M, N, K, fp8, kw):
    got, want = _gemm_case(qb, M, N, K, fp8=fp8, seed=M, **kw)
    _check_gemm(got, want, f"gemm {M}x{N}x{K} fp8={fp8} {kw}", fp8)
    again, _ = _gemm_case(qb, M, N, K, fp8=fp8, seed=M, **kw)
    np.testing.assert_array_equal(got.to_numpy(), again.to_numpy())


def test_tensor_maps_of_many_geometries_and_addresses(qb):
    """The maps kept are those of geometries: more of them than are kept, each with tensors at two addresses in turn."""
    from oracle import ops
    from tests import util
    from tests.test_gpu_kernels import T

    r = util.rng(97)
    shapes = [(8 * i, 64 + 16 * (i % 7)) for i in range(1, 81)]
    pairs = [[(util.bf16_randn(r, (5, K)), util.bf16_randn(r, (N, K))) for _ in range(2)] for N, K in shapes]
    dev = [[(T(qb, a, "bf16"), T(qb, b, "bf16")) for a, b in two] for two in pairs]
    for which in (0, 1, 0):
        for two, d in zip(pairs, dev):
            got = qb.qf.gemm(*d[which], out_dtype="f32", split_k=1)
            _check_gemm(got, ops.gemm(*two[which], return_f32=True), f"{two[which][1].shape} {which}", False)

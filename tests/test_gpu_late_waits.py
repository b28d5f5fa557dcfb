"""What the kernels leave of a call in which a wait ran out: the rows that the late work belongs to stay as they were, in every CTA that
would have written a part of them, all others are what they always are, and the status says so.

The library is built once more with QB_LATE_WAIT (``late`` in csrc/sm100.cuh): the MMA thread of the last CTAs of a grid, all its work
done, waits half a millisecond for a flag that nothing sets and gives up.  A child process loads it and makes the calls below."""

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

pytestmark = pytest.mark.gpu

MARK = 0x7FC1  # a bf16 NaN that no call computes


def attention(kv_dt, H, W, Hk, gqa, nb, splits):
    """Packed output [tokens, heads, 64]; whether the tickets were left at zero."""

    def run(qb):
        from oracle import ops
        from tests import util
        from tests.test_gpu_kernels import T

        r = util.rng([90, H, Hk])
        tpf, Hq = H * W, Hk * gqa
        cap = (nb + 1) * tpf
        make = util.bf16_randn if kv_dt == "bf16" else util.e4m3_randn
        segs, n = ops.compute_segments(1000, nb, tpf, 1)
        out = T(qb, np.full((tpf, Hq * 64), MARK, np.uint16), "bf16")
        qb.qf.owl_attn(T(qb, util.bf16_randn(r, (tpf, (Hq + 2 * Hk) * 64)), "bf16"), T(qb, make(r, (Hk * cap, 64)), kv_dt), T(qb, make(r, (Hk * 64, cap)), kv_dt),
                       T(qb, np.asarray(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, Hk, gqa, H, W, nb, 1, compute_dtype=kv_dt, packed_qkv=True,
                       frame_t=T(qb, np.array([1000], np.int32)), out=out, kv_splits=splits)  # fmt: skip
        ws = qb.functional._ATTN_WS
        return out.to_numpy().reshape(tpf, Hq, 64), ws is None or not ws.to_numpy()[: 16 << 10].any()

    return run


def product(fp8, M, N, K, **kw):
    """The result; whether the tile counters were left at zero."""

    def run(qb):
        from tests import util
        from tests.test_gpu_kernels import T

        r, dt = util.rng([91, M, N]), "e4m3" if fp8 else "bf16"
        make = util.e4m3_randn if fp8 else util.bf16_randn
        out = T(qb, np.full((M, N), MARK, np.uint16), "bf16")
        gate = dict(gate=T(qb, util.bf16_randn(r, (1, N)), "bf16"), residual=T(qb, util.bf16_randn(r, (M, N)), "bf16"))
        qb.qf.gemm(T(qb, make(r, (M, K)), dt), T(qb, make(r, (N, K), 0.05), dt), out=out, **gate, **kw)
        ws = qb.functional._WS
        return out.to_numpy(), ws is None or not ws.to_numpy()[: 64 << 10].any()

    return run


def projection(qb):
    """The QKV projection with its epilogue, four K slices a tile (2 Q heads, 1 KV head, 128 tokens)."""
    from tests import util
    from tests.test_gpu_kernels import T

    r, i32 = util.rng(92), lambda *v: T(qb, np.array(v, np.int32))
    out = T(qb, np.full((128, 256), MARK, np.uint16), "bf16")
    qb.qf.gemm_qkv_post(T(qb, util.bf16_randn(r, (128, 2048)), "bf16"), T(qb, util.bf16_randn(r, (256, 2048), 0.05), "bf16"), None, None, i32(3), i32(0),
                        T(qb, np.zeros((64, 640), np.uint16), "bf16"), i32(0, 0, 0, 0, 0, 0), i32(0), T(qb, np.zeros((640, 64), np.uint16), "bf16"),
                        n_q_heads=2, n_kv_heads=1, H_spatial=16, W_spatial=8, num_buckets=4, pinned_dilation=1, out=out)  # fmt: skip
    return out.to_numpy(), True


def grouped(qb):
    from tests import util
    from tests.test_gpu_kernels import T

    r = util.rng(93)
    out = T(qb, np.full((512, 64), MARK, np.uint16), "bf16")
    qb.qf.gemm_grouped(T(qb, util.bf16_randn(r, (512, 512)), "bf16"), T(qb, util.bf16_randn(r, (128, 512), 0.05), "bf16"), T(qb, np.array([0, 0, 0, 1], np.int32)),
                       n_experts=2, out=out)  # fmt: skip
    return out.to_numpy(), True


# name -> (call, which part of its result is late)
LAST_QUERY_TILE, LAST_HEAD = np.s_[128:], np.s_[:, 47:]
CASES = {
    f"attention {kv_dt} {name}": (attention(kv_dt, 16, 16, Hk, 2, nb, splits), late)
    for kv_dt in ("bf16", "e4m3")
    for name, Hk, nb, splits, late in [
        ("one CTA an item", 1, 8, 1, LAST_QUERY_TILE),
        ("cluster of 2", 1, 8, 2, LAST_QUERY_TILE),
        ("cluster of 7", 1, 16, 7, LAST_QUERY_TILE),
        ("9 parts through the workspace", 1, 16, 9, LAST_QUERY_TILE),
        ("helpers", 24, 64, 0, LAST_HEAD),  # 96 items, 52 helpers: the last takes the two query tiles of head 47
    ]
}
CASES.update({
    f"gemm {'e4m3' if fp8 else 'bf16'} {name}": (product(fp8, M, N, K, **kw), late)
    for fp8 in (False, True)
    for name, M, N, K, kw, late in [
        ("one slice", 200, 192, 512, dict(split_k=1, tile_n=64), np.s_[:, 128:]),
        ("one slice, column remainder", 200, 200, 512, dict(split_k=1, tile_n=128), np.s_[:, 128:]),
        ("cluster of 4 slices", 200, 192, 2048, dict(split_k=4, tile_n=64), np.s_[:, 128:]),
        ("3 slices through the workspace", 200, 192, 2048, dict(split_k=3, tile_n=64, slice_mode=1), np.s_[:, 128:]),
        ("pairs", 1700, 1800, 4096 if fp8 else 2048, dict(), np.s_[1536:, 1792:]),
        ("pairs, 2 slices", 300, 2048, 8192, dict(split_k=2, tile_n=128), np.s_[256:, 1920:]),
    ]
})
CASES["qkv projection, cluster of 4 slices"] = projection, np.s_[:, 192:]
CASES["grouped"] = grouped, np.s_[:]


def run_all(qb):
    results = {}
    for name, (call, _) in CASES.items():
        qb._lib.device_status()
        results[name], results[name + " tickets"] = call(qb)
        results[name + " status"] = qb._lib.device_status()
    return results


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    import quark_b200 as qb

    qb._lib.require_device(0)
    tmp = tmp_path_factory.mktemp("late")
    env = dict(os.environ, QB_BUILD_DIR=str(tmp), QB_BUILD_FLAGS="-DQB_LATE_WAIT")
    subprocess.run(["bash", str(ROOT / "quark_b200/csrc/build.sh")], env=env, check=True, timeout=600)
    env = dict(os.environ, QUARK_B200_LIB_PATH=str(tmp / "libquark_b200.so"))
    subprocess.run([sys.executable, __file__, str(tmp / "late.npz")], env=env, check=True, timeout=300)
    return run_all(qb), np.load(tmp / "late.npz")


@pytest.mark.parametrize("name", list(CASES))
def test_rows_of_late_work_stay_as_they_were(results, name):
    usual, late = results
    assert usual[name + " status"] == 0 and late[name + " status"] != 0
    assert not (usual[name] == MARK).any()
    want = usual[name].copy()
    want[CASES[name][1]] = MARK
    np.testing.assert_array_equal(late[name], want)
    assert usual[name + " tickets"] and late[name + " tickets"]


if __name__ == "__main__":
    import quark_b200

    np.savez(sys.argv[1], **run_all(quark_b200))

"""The branches that a call's sizes choose: key shares of the attention, expert runs of the routing and of the grouped GEMM, column
remainders of the GEMM epilogues, the captured append pass, and the calls that are checked and made in C."""

import dataclasses

import numpy as np
import pytest

from oracle import codec, ops
from tests import util
from tests.test_gpu_kernels import T, _attn_check, _check_gemm, _gemm_case
from tests.util import bf16_randn, e4m3_randn, f32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qb():
    import quark_b200 as q

    q._lib.require_device(0)
    yield q
    q.runtime.synchronize()
    assert q._lib.device_status() == 0


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("H,W,Hk,gqa,nb,ft", [
    (4, 16, 1, 1, 40, 60),  # one query tile, half of it empty: the widest sharing
    (16, 8, 2, 1, 6, 3),  # fewer buckets than a cluster has CTAs
    (12, 20, 3, 2, 5, 30),  # a second query tile of 112 rows, key tiles that end inside a share
    (16, 16, 5, 2, 9, 100),
    (16, 8, 8, 4, 16, 100),
    (8, 18, 16, 2, 3, 9),  # more items than clusters fit at once
    (16, 16, 24, 2, 64, 100),  # 96 items and 52 helpers of one or two items
    (16, 16, 24, 2, 64, 2),  # the same before the ring has filled: whole items
    (16, 9, 25, 2, 96, 200),  # keys and queries that end inside a tile
    (20, 16, 43, 1, 100, 200),  # 129 items: helpers of six or seven
])  # fmt: skip
def test_attention_key_shares_by_size(qb, kv_dt, H, W, Hk, gqa, nb, ft):
    r = util.rng([81, H, Hk])
    tpf, cap, Hq = H * W, (nb + 1) * H * W, Hk * gqa
    qkv = ops.head_rmsnorm(bf16_randn(r, (tpf, (Hq + 2 * Hk) * 64)), n_q_heads=Hq, n_kv_heads=Hk)
    make = bf16_randn if kv_dt == "bf16" else e4m3_randn
    Kc, Vc = make(r, (Hk * cap, 64)), make(r, (Hk * 64, cap))
    segs, n = ops.compute_segments(ft, nb, tpf, 1)
    args = (T(qb, qkv, "bf16"), T(qb, Kc, kv_dt), T(qb, Vc, kv_dt), T(qb, np.asarray(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, Hk, gqa, H, W, nb, 1)
    kw = dict(compute_dtype="e4m3" if kv_dt == "e4m3" else None, packed_qkv=True, frame_t=T(qb, np.array([ft], np.int32)))
    want = ops.owl_attn(qkv, Kc, Vc, segs, [n], ft, n_kv_heads=Hk, gqa_ratio=gqa, H_spatial=H, W_spatial=W, kv_dtype=kv_dt,
                        q_quant="e4m3" if kv_dt == "e4m3" else None)  # fmt: skip
    for splits in (0, 1, 3, 8):
        got = qb.qf.owl_attn(*args, kv_splits=splits, **kw).to_numpy()
        _attn_check(got, want, f"attn {H}x{W} Hk={Hk} splits={splits} {kv_dt}", kv_dt == "e4m3")
        np.testing.assert_array_equal(got, qb.qf.owl_attn(*args, kv_splits=splits, **kw).to_numpy())


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("H,W,ft", [
    (8, 8, 0),  # half of one key tile: two of three groups have nothing
    (8, 8, 1),  # two segments in one tile
    (16, 8, 2),  # a tile for each of three groups, an odd number for two
    (16, 8, 3),
    (12, 20, 4),  # nine tiles and a remainder, a query tile of 112 rows
    (17, 16, 5),
])  # fmt: skip
def test_attention_groups_over_tiles_whose_maximum_jumps(qb, kv_dt, H, W, ft):
    """The groups of a CTA, and the CTAs that share an item (clusters of odd size among them), take key tiles in turn; the scores grow
    and shrink from tile to tile by far more than the slack within which a maximum is kept.  Against the oracle fed the rotated
    query as the kernel narrows it, as for scores that drift, with that test's tolerance."""
    r = util.rng([97, H, ft])
    Hk, gqa, nb = 2, 2, 6
    tpf, cap = H * W, (nb + 1) * H * W
    qkv = ops.head_rmsnorm(bf16_randn(r, (tpf, 8 * 64)), n_q_heads=4, n_kv_heads=2)
    step = np.array([0.3, 6.0, 1.0, 14.0, 0.1, 9.0, 13.0], np.float32)[np.arange(cap) // 128 % 7]
    to = codec.f32_to_bf16 if kv_dt == "bf16" else codec.f32_to_e4m3
    Kc = to((r.standard_normal((Hk, cap, 64), dtype=np.float32) * step[None, :, None]).reshape(Hk * cap, 64))
    Vc = to(r.standard_normal((Hk * 64, cap), dtype=np.float32))
    segs, n = ops.compute_segments(ft, nb, tpf, 1)
    with codec.bf16_rounding("rne"):
        want = ops.owl_attn(qkv, Kc, Vc, segs, [n], ft, n_kv_heads=Hk, gqa_ratio=gqa, H_spatial=H, W_spatial=W, kv_dtype=kv_dt, q_quant=kv_dt)
    args = (T(qb, qkv, "bf16"), T(qb, Kc, kv_dt), T(qb, Vc, kv_dt), T(qb, np.asarray(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, Hk, gqa, H, W, nb, 1)
    kw = dict(compute_dtype="e4m3" if kv_dt == "e4m3" else None, packed_qkv=True, frame_t=T(qb, np.array([ft], np.int32)))
    for splits in (1, 2, 3, 5, 7):
        _attn_check(qb.qf.owl_attn(*args, kv_splits=splits, **kw).to_numpy(), want, f"attn {H}x{W} ft={ft} splits={splits} {kv_dt}", kv_dt == "e4m3")


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("H,W,Hk,gqa,nb,ft", [
    (16, 16, 24, 2, 65, 900),  # 96 items on 148 SMs: owners walk 93 tiles, helpers two pieces of 37
    (17, 16, 39, 1, 127, 300),  # 117 items: up to four pieces of 47 a helper, partial tiles of three segments, a query tile of 16 rows
    (17, 16, 43, 1, 101, 300),  # 129 items: up to seven pieces of 19 a helper
])  # fmt: skip
def test_attention_with_helpers_over_tiles_whose_maximum_jumps(qb, kv_dt, H, W, Hk, gqa, nb, ft):
    """The same keys for CTAs that work on one piece of an item after the other, so that a maximum, a barrier phase or a place in the table
    left over from the piece before would show.  The oracle, fed and compared as above, computes the heads of three KV heads."""
    import ctypes as C

    r = util.rng([99, H, Hk])
    tpf, cap, Hq = H * W, (nb + 1) * H * W, Hk * gqa
    dt = qb._lib.DTYPE_CODE[kv_dt]
    p = qb._lib.AttnParams(n_kv_heads=Hk, gqa_ratio=gqa, H_spatial=H, W_spatial=W, num_buckets=nb, pinned_dilation=1, kv_dtype=dt, compute_dtype=dt, max_segments=3,
                           packed_qkv=1, quilt_factor=1)  # fmt: skip
    assert qb._lib.load().qb_owl_attn_scratch_bytes(C.byref(p)) > 0  # there are helpers
    qkv = ops.head_rmsnorm(bf16_randn(r, (tpf, (Hq + 2 * Hk) * 64)), n_q_heads=Hq, n_kv_heads=Hk)
    step = np.array([0.3, 6.0, 1.0, 14.0, 0.1, 9.0, 13.0], np.float32)[np.arange(cap) // 128 % 7]
    to = codec.f32_to_bf16 if kv_dt == "bf16" else codec.f32_to_e4m3
    one = to(r.standard_normal((cap, 64), dtype=np.float32) * step[:, None]), to(r.standard_normal((64, cap), dtype=np.float32))
    turn = [int(t) * 16 for t in r.integers(0, cap // 16, Hk)]  # every head another order of the same keys
    Kc, Vc = np.concatenate([np.roll(one[0], t, 0) for t in turn]), np.concatenate([np.roll(one[1], t, 1) for t in turn])
    segs, n = ops.compute_segments(ft, nb, tpf, 1)
    got = qb.qf.owl_attn(T(qb, qkv, "bf16"), T(qb, Kc, kv_dt), T(qb, Vc, kv_dt), T(qb, np.asarray(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, Hk, gqa, H, W, nb, 1,
                         compute_dtype=kv_dt, packed_qkv=True, frame_t=T(qb, np.array([ft], np.int32))).to_numpy().reshape(tpf, Hq, 64)  # fmt: skip
    heads = qkv.reshape(tpf, Hq + 2 * Hk, 64)
    for h in (0, Hk // 2, Hk - 1):
        mine = np.concatenate([heads[:, h * gqa : (h + 1) * gqa], heads[:, Hq + h : Hq + h + 1], heads[:, Hq + Hk + h : Hq + Hk + h + 1]], 1).reshape(tpf, -1)
        with codec.bf16_rounding("rne"):
            want = ops.owl_attn(mine, Kc[h * cap : (h + 1) * cap], Vc[h * 64 : (h + 1) * 64], segs, [n], ft, n_kv_heads=1, gqa_ratio=gqa, H_spatial=H, W_spatial=W,
                                kv_dtype=kv_dt, q_quant=kv_dt)  # fmt: skip
        _attn_check(np.ascontiguousarray(got[:, h * gqa : (h + 1) * gqa]).reshape(tpf, -1), want, f"helpers {H}x{W} head {h} {kv_dt}", kv_dt == "e4m3")


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("Hk,nb", [(1, 16), (24, 64)])  # key splits in clusters, one CTA per item (helpers want a workspace)
def test_attention_call_without_a_workspace(qb, kv_dt, Hk, nb):
    import ctypes as C

    lib, r = qb._lib.load(), util.rng([96, Hk])
    segs, n = ops.compute_segments(500, nb, 256, 1)
    make = bf16_randn if kv_dt == "bf16" else e4m3_randn
    qkv, K, V = T(qb, bf16_randn(r, (256, Hk * 4 * 64)), "bf16"), T(qb, make(r, (Hk * (nb + 1) * 256, 64)), kv_dt), T(qb, make(r, (Hk * 64, (nb + 1) * 256)), kv_dt)
    seg, nseg, ft = T(qb, np.array(segs, np.int32)), T(qb, np.array([n], np.int32)), T(qb, np.array([500], np.int32))
    want = qb.qf.owl_attn(qkv, K, V, seg, nseg, 1, Hk, 2, 16, 16, nb, 1, compute_dtype=kv_dt, packed_qkv=True, frame_t=ft, kv_splits=0 if Hk == 1 else 1).to_numpy()
    out = T(qb, np.zeros(want.shape, np.uint16), "bf16")
    dt = qb._lib.DTYPE_CODE[kv_dt]
    p = qb._lib.AttnParams(n_kv_heads=Hk, gqa_ratio=2, H_spatial=16, W_spatial=16, num_buckets=nb, pinned_dilation=1, kv_dtype=dt, compute_dtype=dt, max_segments=3,
                           packed_qkv=1, quilt_factor=1)  # fmt: skip
    qb._lib.check(lib.qb_owl_attn(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), seg.data_ptr(), nseg.data_ptr(), ft.data_ptr(), out.data_ptr(), None,
                                  qb.qf.rope_table(16, 16).data_ptr(), C.byref(p), None, 0, qb.runtime.active_stream()))  # fmt: skip
    np.testing.assert_array_equal(out.to_numpy(), want)


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
@pytest.mark.parametrize("Hk,nb", [(1, 16), (24, 64)])  # key splits in clusters, one CTA per item
def test_attention_reads_the_table_that_the_kernel_before_it_builds(qb, kv_dt, Hk, nb):
    """A caller's table made on the device by the call just before, where another grid's table stood: the angles of the finished one."""
    import ctypes as C

    lib, r, stream = qb._lib.load(), util.rng([94, Hk]), qb.runtime.active_stream()
    H, W = 8, 32
    segs, n = ops.compute_segments(500, nb, 256, 1)
    make = bf16_randn if kv_dt == "bf16" else e4m3_randn
    qkv, K, V = T(qb, bf16_randn(r, (256, Hk * 4 * 64)), "bf16"), T(qb, make(r, (Hk * (nb + 1) * 256, 64)), kv_dt), T(qb, make(r, (Hk * 64, (nb + 1) * 256)), kv_dt)
    seg, nseg, ft = T(qb, np.array(segs, np.int32)), T(qb, np.array([n], np.int32)), T(qb, np.array([500], np.int32))
    table = qb.QuarkTensor.empty(256, 16, dtype="f32")
    dt = qb._lib.DTYPE_CODE[kv_dt]
    p = qb._lib.AttnParams(n_kv_heads=Hk, gqa_ratio=2, H_spatial=H, W_spatial=W, num_buckets=nb, pinned_dilation=1, kv_dtype=dt, compute_dtype=dt, max_segments=3,
                           packed_qkv=1, quilt_factor=1)  # fmt: skip

    def attend(out):
        qb._lib.check(lib.qb_owl_attn(qkv.data_ptr(), K.data_ptr(), V.data_ptr(), seg.data_ptr(), nseg.data_ptr(), ft.data_ptr(), out.data_ptr(), None,
                                      table.data_ptr(), C.byref(p), None, 0, stream))  # fmt: skip

    def build(h, w):
        qb._lib.check(lib.qb_rope_table_build(table.data_ptr(), h, w, stream))

    outs = [T(qb, np.zeros((256, Hk * 2 * 64), np.uint16), "bf16") for _ in range(12)]
    build(H, W)
    qb.runtime.synchronize()
    attend(outs[0])
    build(W, H)
    qb.runtime.synchronize()
    attend(outs[1])
    for out in outs[2:]:
        build(W, H)
        build(H, W)
        attend(out)
    got = [o.to_numpy() for o in outs]
    assert (got[0] != got[1]).any()
    for g in got[2:]:
        np.testing.assert_array_equal(g, got[0])


@pytest.mark.parametrize("kv_dt", ["bf16", "e4m3"])
def test_attention_with_helpers_does_not_depend_on_who_comes_last(qb, kv_dt):
    """The two parts of an item are summed by the CTA that finishes second.  A product on another stream keeps 100 SMs for about 100 us,
    so that the helpers, the last CTAs of the grid, start late: the same bits as alone."""
    import ctypes as C

    lib, stream, r = qb._lib.load(), qb.runtime.stream, util.rng(95)
    make = bf16_randn if kv_dt == "bf16" else e4m3_randn
    segs, n = ops.compute_segments(500, 64, 256, 1)
    args = (T(qb, bf16_randn(r, (256, 96 * 64)), "bf16"), T(qb, make(r, (24 * 65 * 256, 64)), kv_dt), T(qb, make(r, (24 * 64, 65 * 256)), kv_dt),
            T(qb, np.array(segs, np.int32)), T(qb, np.array([n], np.int32)), 1, 24, 2, 16, 16, 64, 1)  # fmt: skip
    kw = dict(compute_dtype=kv_dt, packed_qkv=True, frame_t=T(qb, np.array([500], np.int32)))
    want = qb.qf.owl_attn(*args, **kw).to_numpy()
    outs = [T(qb, np.zeros(want.shape, np.uint16), "bf16") for _ in range(10)]
    a, c = qb.QuarkTensor.zeros(1280, 32768, dtype="bf16"), qb.QuarkTensor.zeros(1280, 1280, dtype="bf16")
    p, first = C.c_void_p(), qb.runtime.active_stream()
    qb._lib.check(lib.qb_stream_create(C.byref(p)))
    try:
        for out in outs:
            qb._lib.check(lib.qb_device_sync())
            stream.set_stream(int(p.value))
            qb.qf.gemm(a, a, out=c, split_k=1, tile_n=128)
            stream.set_stream(first)
            qb.qf.owl_attn(*args, out=out, **kw)
    finally:
        stream.set_stream(first)
        qb._lib.check(lib.qb_device_sync())
    for out in outs:
        np.testing.assert_array_equal(out.to_numpy(), want)
    qb._lib.check(lib.qb_stream_destroy(p))


def test_attention_with_helpers_on_two_streams_and_in_a_graph(qb):
    """The helpers' partial results and tickets lie in a workspace: calls that overlap, eager on two streams and replayed from a graph,
    each have one, and every result is that of a call alone."""
    import ctypes as C

    lib, stream, r = qb._lib.load(), qb.runtime.stream, util.rng(94)
    H = W = 16
    Hk, nb = 24, 64
    calls = []
    for i in range(3):
        args = (T(qb, bf16_randn(r, (256, 96 * 64)), "bf16"), T(qb, e4m3_randn(r, (Hk * 65 * 256, 64)), "e4m3"), T(qb, e4m3_randn(r, (Hk * 64, 65 * 256)), "e4m3"),
                T(qb, np.array(ops.compute_segments(500, nb, 256, 1)[0], np.int32)), T(qb, np.array([ops.compute_segments(500, nb, 256, 1)[1]], np.int32)))  # fmt: skip
        out, ft = T(qb, np.zeros((256, 48 * 64), np.uint16), "bf16"), T(qb, np.array([500], np.int32))
        calls.append((lambda a=args, o=out, f=ft: qb.qf.owl_attn(*a, 1, Hk, 2, H, W, nb, 1, compute_dtype="e4m3", packed_qkv=True, frame_t=f, out=o), out))
    want = []
    for call, out in calls:
        call()
        want.append(out.to_numpy())
        out.zero_()
    cap = qb.runtime.capture_graph()
    with cap:
        calls[2][0]()
    qb.runtime.synchronize()
    first, handles = qb.runtime.active_stream(), []
    for _ in range(2):
        p = C.c_void_p()
        qb._lib.check(lib.qb_stream_create(C.byref(p)))
        handles.append(int(p.value))
    try:
        for _ in range(20):  # in turn, so that the streams' queues run side by side
            for handle, run in zip([first, *handles], (calls[0][0], calls[1][0], cap.graph.launch)):
                stream.set_stream(handle)
                run()
    finally:
        stream.set_stream(first)
        qb._lib.check(lib.qb_device_sync())
    for (_, out), w in zip(calls, want):
        np.testing.assert_array_equal(out.to_numpy(), w)
    assert len({id(t) for t in (qb.functional._ATTN_WS, cap.graph.scratch[1], qb.functional._OF_STREAM[handles[0]][1])}) == 3
    for handle in handles:
        qb.functional._OF_STREAM.pop(handle, None)
        qb._lib.check(lib.qb_stream_destroy(C.c_void_p(handle)))


@pytest.mark.parametrize("M,E,K", [(1, 8, 2), (1025, 8, 4), (2500, 32, 3), (4096, 24, 2)])
def test_routing_by_size(qb, M, E, K):
    r = util.rng([82, M])
    logits = bf16_randn(r, (M, E))
    n = qb.qf.moe_slots(M, E, K)
    got = [t.to_numpy().reshape(-1) for t in qb.qf.moe_route_slots(T(qb, logits, "bf16"), top_k=K)]
    want = ops.moe_route_slots(logits, K, tile=128, total_slots=n)
    for g, key in zip(got, ("slot_token", "slot_weight", "tile_expert", "token_slot")):
        if key == "slot_weight":
            np.testing.assert_allclose(g, want[key], atol=1e-6)
        else:
            np.testing.assert_array_equal(g, want[key].reshape(-1))


@pytest.mark.parametrize("D", [16, 72 * 16])
def test_gather_narrows_as_quantize_does(qb, D):
    r = util.rng(83)
    x = T(qb, bf16_randn(r, (100, D)), "bf16")
    st = np.full(256, -1, np.int32)
    st[:90] = r.permutation(100)[:90]
    out = qb.qf.moe_gather(x, T(qb, st), out=T(qb, np.full((256, D), 0x7F, np.uint8), "e4m3")).to_numpy()
    np.testing.assert_array_equal(out[:90], qb.qf.quantize_e4m3(x).to_numpy()[st[:90]])
    assert not out[90:].any()


@pytest.mark.parametrize("fp8", [False, True])
def test_dense_experts_take_the_k_slices_of_their_products(qb, fp8):
    """The dense schedule is one product after the other as ``qf.gemm`` plans them (a few slices each at this size)."""
    from quark_b200 import nn as qnn

    r, qf = util.rng([98, fp8]), qb.qf
    M, D, H, E = 128, 1024, 2048, 8
    layer = {s: qnn.MoE(M, D, H, E, 2, schedule=s) for s in ("dense", "sorted")}
    weights = [T(qb, bf16_randn(r, shape, std), "bf16") for shape, std in (((E, D), 0.2), ((E * H, D), 0.05), ((E * D, H), 0.05))]
    for m in layer.values():
        m.router.weight.data, m.expert_in.data, m.expert_out.data = weights
        m.prepare(fp8=fp8)
    x = T(qb, bf16_randn(r, (M, D)), "bf16")
    dense, w_in, w_out = layer["dense"], layer["dense"].expert_in.data, layer["dense"].expert_out.data
    got = dense(x).to_numpy()
    partials = T(qb, np.zeros((E * M, D), np.float32))
    for e in range(E):
        h = qf.gemm(qf.quantize_e4m3(x) if fp8 else x, w_in.rows(e * H, (e + 1) * H), activation="silu")
        qf.gemm(h, w_out.rows(e * D, (e + 1) * D), out_dtype="f32", out=partials.rows(e * M, (e + 1) * M))
    np.testing.assert_array_equal(qf.moe_combine(partials, qf.moe_route(dense.router(x), top_k=2)).to_numpy(), got)
    # the sorted schedule's sums are in another order; a hidden value on the edge of two codes may take the other
    g, s = f32(got, "bf16"), f32(layer["sorted"](x).to_numpy(), "bf16")
    assert np.linalg.norm(g - s) <= (2e-2 if fp8 else 6e-3) * np.linalg.norm(g)


@pytest.mark.parametrize("runs,N,K", [
    ([1, 0, 0], 64, 64),  # one tile of one expert
    ([3, 1, 2], 328, 192),  # odd numbers of tiles, columns that end inside a tile
    ([2, 5, 0, 4], 1032, 2064),  # a K remainder
])  # fmt: skip
@pytest.mark.parametrize("fp8", [False, True])
def test_grouped_gemm_by_expert_runs(qb, fp8, runs, N, K):
    r = util.rng([84, N])
    tiles = np.concatenate([np.full(c, e) for e, c in enumerate(runs)] + [[-1, -1]]).astype(np.int32)
    E, M, dt = len(runs), 128 * len(tiles), "e4m3" if fp8 else "bf16"
    A = e4m3_randn(r, (M, K)) if fp8 else bf16_randn(r, (M, K))
    B = e4m3_randn(r, (E * N, K), 0.05) if fp8 else bf16_randn(r, (E * N, K), 0.05)
    a, b, t = T(qb, A, dt), T(qb, B, dt), T(qb, tiles)
    got = qb.qf.gemm_grouped(a, b, t, n_experts=E, activation="silu", compute_dtype=dt, out=T(qb, np.zeros((M, N), np.uint16), "bf16"))
    g = got.to_numpy()
    for i, e in enumerate(tiles[tiles >= 0]):
        rows = slice(128 * i, 128 * i + 128)
        want = ops.gemm(A[rows], B[e * N : (e + 1) * N], a_dtype=dt, b_dtype=dt, activation="silu", return_f32=True)
        _check_gemm(T(qb, g[rows], "bf16"), want, f"tile {i} expert {e} fp8={fp8}", fp8)
    # an e4m3 result through bf16 is the bf16 result narrowed
    q = qb.qf.gemm_grouped(a, b, t, n_experts=E, activation="silu", compute_dtype=dt, out_dtype="e4m3", through_bf16=True,
                           out=T(qb, np.zeros((M, N), np.uint8), "e4m3"))  # fmt: skip
    np.testing.assert_array_equal(q.to_numpy(), qb.qf.quantize_e4m3(got).to_numpy())


@pytest.mark.parametrize("M,N,kw", [
    (1, 8, dict()),
    (5, 72, dict(gate_groups=5)),
    (130, 88, dict(gate_groups=2)),
    (130, 152, dict(out_dtype="f32", bias=True)),
    (200, 200, dict(out_dtype="e4m3", act="silu", bias=True)),
    (260, 1000, dict(gate_groups=4)),
])  # fmt: skip
@pytest.mark.parametrize("fp8", [False, True])
def test_epilogue_of_column_remainders(qb, M, N, kw, fp8):
    got, want = _gemm_case(qb, M, N, 272, fp8=fp8, seed=M + N, split_k=1, **kw)
    _check_gemm(got, want, f"{M}x{N} {kw} fp8={fp8}", fp8)


@pytest.mark.parametrize("quant", ["bf16", "fp8"])
def test_append_pass_captured_equals_call_by_call(qb, quant):
    from quark_b200.models import QuantConfig, Waypoint15Config, make_params

    q = QuantConfig.all_fp8() if quant == "fp8" else QuantConfig.all_bf16()
    cfg = Waypoint15Config(d_model=128, n_layers=4, n_heads=2, n_kv_heads=1, height=8, width=8, channels=4, local_window=2, global_window=4,
                           global_pinned_dilation=2, quant=q)  # fmt: skip
    params = make_params(cfg, seed=5, weight_std=0.08)
    r = util.rng(85)
    engines = [qb.Engine(cfg=cfg, quant=q, params=params, use_graph=g) for g in (True, False)]
    for i in range(6):
        lat = codec.f32_to_bf16(r.standard_normal((1, cfg.latent_numel)).astype(np.float32))
        for e in engines:
            if i == 4:  # a parameter replaced after the capture has to be seen by the next append
                p = dict(e.model.named_parameters())
                name = next(k for k, v in p.items() if v.data.dtype == "bf16" and v.data.ndim == 2 and "weight" in k)
                p[name].data = T(qb, np.zeros_like(p[name].data.to_numpy()), "bf16")
            e.append_frame(lat)
        for a, b in zip(engines[0].model.blocks, engines[1].model.blocks):
            for x in ("K_cache", "Vt_cache", "segments", "n_segments"):
                np.testing.assert_array_equal(getattr(a.kv_cache, x).to_numpy(), getattr(b.kv_cache, x).to_numpy())


def _new_caches(qb, e):
    kc = e.model.blocks[1].kv_cache
    new = qb.nn.KVCacheUpdate(rope_n_frames=1, Dh=64, dtype=kc.K_cache.dtype, **kc._kw)
    for k in ("K_cache", "Vt_cache", "segments", "n_segments"):
        getattr(new, k).copy_from(getattr(kc, k))
    e.model.blocks[1].kv_cache = new


def _host_side_of_its_own(qb, e):
    blk, own = e.model.blocks[1], e.model.blocks[1].forward
    e.seen = []
    blk.forward = lambda *a, **kw: (e.seen.append(1), own(*a, **kw))[1]


def _new_lut_row(qb, e):
    lut = e.model.blocks[1]._cond_lut
    lut[-1] = tuple(T(qb, np.zeros(t.shape, np.uint16), "bf16") for t in lut[-1])


def _new_counter(qb, e):
    e.gen.frame_t = T(qb, e.gen.frame_t.to_numpy() + 3)


@pytest.mark.parametrize("change", [
    _new_caches,
    _host_side_of_its_own,
    _new_lut_row,
    _new_counter,
    lambda qb, e: setattr(e.model.blocks[1].qkv_proj, "w_scale", T(qb, np.linspace(0.5, 2.0, e.cfg.qkv_dim, dtype=np.float32))),
    lambda qb, e: e.model.blocks[1].kv_cache.set_scales(np.full(1, 2.0, np.float32), np.full(1, 0.5, np.float32)),
    lambda qb, e: setattr(e.model.blocks[1], "mlp", e.model.blocks[2].mlp),
    lambda qb, e: setattr(e.model.blocks[1], "_cfg", dataclasses.replace(e.cfg, fuse_gate_residual=False)),
])  # fmt: skip
def test_append_pass_captured_follows_a_changed_model(qb, change):
    """Whatever a pass reads of the model and of the engine, changed after the capture, is seen by the next append."""
    from quark_b200.models import QuantConfig, Waypoint15Config, make_params

    q = QuantConfig(linear="fp8", kv_cache="fp8", attn_compute="bf16")  # the attention reads shadow caches
    cfg = Waypoint15Config(d_model=128, n_layers=3, n_heads=2, n_kv_heads=1, height=8, width=8, channels=4, local_window=2, global_window=4,
                           global_pinned_dilation=2, quant=q)  # fmt: skip
    params = make_params(cfg, seed=9, weight_std=0.08)
    r = util.rng(88)
    engines = [qb.Engine(cfg=cfg, quant=q, params=params, use_graph=g) for g in (True, False)]
    for i in range(7):
        lat = codec.f32_to_bf16(r.standard_normal((1, cfg.latent_numel)).astype(np.float32))
        for e in engines:
            if i == 3:
                change(qb, e)
            e.append_frame(lat)
        for a, b in zip(engines[0].model.blocks, engines[1].model.blocks):
            for x in ("K_cache", "Vt_cache", "segments", "n_segments"):
                np.testing.assert_array_equal(getattr(a.kv_cache, x).to_numpy(), getattr(b.kv_cache, x).to_numpy(), err_msg=f"append {i}")
    if change is _host_side_of_its_own:
        assert len(engines[0].seen) == len(engines[1].seen) == 4
    else:
        assert engines[0]._append_graph._graph is not None  # captured again


@pytest.mark.parametrize("use_graph", [True, False])
def test_shadow_caches_follow_replaced_caches(qb, use_graph):
    """Caches put in the place of others are brought over whole, however often either was written from the host."""
    from quark_b200.models import QuantConfig, Waypoint15Config, make_params

    q = QuantConfig(linear="fp8", kv_cache="fp8", attn_compute="bf16")
    cfg = Waypoint15Config(d_model=128, n_layers=2, n_heads=2, n_kv_heads=1, height=8, width=8, channels=4, local_window=2, global_window=4,
                           global_pinned_dilation=2, quant=q)  # fmt: skip
    eng, r = qb.Engine(cfg=cfg, quant=q, params=make_params(cfg, seed=9, weight_std=0.08), use_graph=use_graph), util.rng(89)
    kc = eng.model.blocks[0].kv_cache
    for i in range(4):
        if i == 2:
            for name in ("K_cache", "Vt_cache"):
                old = getattr(kc, name)
                new = T(qb, e4m3_randn(r, old.shape), "e4m3")
                new._storage.host_writes = old._storage.host_writes
                setattr(kc, name, new)
        eng.append_frame(codec.f32_to_bf16(r.standard_normal((1, cfg.latent_numel)).astype(np.float32)))
        for cache, sh in zip((kc.K_cache, kc.Vt_cache), kc._shadow):
            np.testing.assert_array_equal(f32(sh.to_numpy(), "bf16"), f32(cache.to_numpy(), "e4m3"), err_msg=f"append {i}")


@pytest.mark.parametrize("quant", ["bf16", "fp8"])
def test_weights_fetched_ahead_change_no_bit(qb, quant, monkeypatch):
    from quark_b200.models import QuantConfig, Waypoint15Config, make_params, waypoint_15

    q = QuantConfig.all_fp8() if quant == "fp8" else QuantConfig.all_bf16()
    cfg = Waypoint15Config(d_model=128, n_layers=3, n_heads=2, n_kv_heads=1, height=8, width=8, channels=4, local_window=2, global_window=4,
                           global_pinned_dilation=2, quant=q)  # fmt: skip
    params = make_params(cfg, seed=7, weight_std=0.08)
    frames = []
    for least in (1 << 62, 0):  # never, always
        monkeypatch.setattr(waypoint_15, "PREFETCH_MIN_BYTES", least)
        eng, r = qb.Engine(cfg=cfg, quant=q, params=params), util.rng(87)
        for _ in range(3):
            eng.append_frame(codec.f32_to_bf16(r.standard_normal((1, cfg.latent_numel)).astype(np.float32)))
        frames.append([eng.gen_frame(noise=r.standard_normal((1, cfg.latent_numel)).astype(np.float32)) for _ in range(3)])
        assert (eng.model._side is not None) == (least == 0)
    for a, b in zip(*frames):
        np.testing.assert_array_equal(a, b)


def test_calls_made_in_c_equal_the_python_path(qb, monkeypatch):
    """Same bytes with and without the extension, and the Python path's errors for what it does not take."""
    qf, r = qb.qf, util.rng(86)
    assert not isinstance(qf._fast, qb._lib._NoFastcall)
    x, y, lat = (T(qb, bf16_randn(r, (24, 256)), "bf16") for _ in range(3))
    row = T(qb, bf16_randn(r, (3, 256)), "bf16")
    w, wq = T(qb, bf16_randn(r, (72, 256)), "bf16"), T(qb, e4m3_randn(r, (72, 256)), "e4m3")
    g72, r72, dsig = T(qb, bf16_randn(r, (3, 72)), "bf16"), T(qb, bf16_randn(r, (24, 72)), "bf16"), T(qb, np.array([0.3], np.float32))
    e = lambda *s, dt="bf16": T(qb, np.zeros(s, {"bf16": np.uint16, "e4m3": np.uint8, "f32": np.float32}[dt]), dt)  # noqa: E731
    calls = [
        lambda: qf.gemm(x, w, out=e(24, 72)),
        lambda: qf.gemm(x, wq, out=e(24, 72, dt="f32"), activation="silu", split_k=2, slice_mode=1),
        lambda: qf.gemm(x, w, gate=g72, residual=r72, gate_groups=3, out=e(24, 72), b_constant=True),
        lambda: qf.ada_rmsnorm(x, row, row, out=e(24, 256)),
        lambda: qf.ada_rmsnorm(x, row, row, 1e-5, "silu", out_q=e(24, 256, dt="e4m3"), only_q=True),
        lambda: qf.rmsnorm(x, out=e(24, 256)),
        lambda: qf.head_rmsnorm(x, 2, 1, 64, out=e(24, 256)),
        lambda: qf.ada_gate_residual(x, y, row, out=e(24, 256)),
        lambda: qf.silu(x, out=e(24, 256), out_q=e(24, 256, dt="e4m3")),
        lambda: qf.add(x, y, out=e(24, 256)),
        lambda: qf.euler_step(x, y, dsig, out=e(24, 256)),
        lambda: qf.quantize_e4m3(x, out=e(24, 256, dt="e4m3")),
        lambda: qf.dequantize_e4m3(wq, out=e(72, 256)),
    ]
    geo = dict(B=1, n_kv_heads=2, H_spatial=8, W_spatial=8, num_buckets=3, pinned_dilation=1)
    hk, hv, hq = (T(qb, bf16_randn(r, (n * 64, 64)), "bf16") for n in (2, 2, 4))
    pk = T(qb, bf16_randn(r, (64, 8 * 64)), "bf16")
    ft, fz = T(qb, np.array([5], np.int32)), T(qb, np.array([0], np.int32))

    def attend(packed, dt, **kw):
        Kc, Vc = T(qb, np.zeros((512, 64), np.uint16 if dt == "bf16" else np.uint8), dt), T(qb, np.zeros((128, 256), np.uint16 if dt == "bf16" else np.uint8), dt)
        seg, nseg = T(qb, np.zeros(6, np.int32)), T(qb, np.zeros(1, np.int32))
        for i in range(4):
            ft.copy_from_numpy(np.array([i], np.int32))
            qf.kv_cache_update(pk if packed else hk, None if packed else hv, ft, fz, Vc, seg, nseg, Kc, packed_qkv=packed, n_q_heads=4, **geo)
        return qf.owl_attn(pk if packed else hq, Kc, Vc, seg, nseg, gqa_ratio=2, packed_qkv=packed, frame_t=ft,
                           **{**geo, "compute_dtype": dt, "out": e(64 if packed else 256, 256 if packed else 64), **kw})  # fmt: skip

    calls += [lambda: attend(False, "bf16"), lambda: attend(True, "e4m3"), lambda: attend(False, "e4m3", kv_splits=2, out_q=e(256, 64, dt="e4m3"))]
    wrong = [
        (ValueError, lambda: attend(False, "bf16", quilt_factor=3)),
        (ValueError, lambda: attend(False, "bf16", out=e(64, 64))),
        (NotImplementedError, lambda: attend(True, "bf16", B=2)),
        (ValueError, lambda: qf.gemm(x, w, out=e(24, 64))),
        (ValueError, lambda: qf.gemm(x, w, out=e(24, 72), out_dtype="f32")),
        (ValueError, lambda: qf.gemm(x, w, out=e(24, 72), gate=g72)),
        (ValueError, lambda: qf.gemm(x, w, out=e(24, 72), gate=g72, residual=r72, gate_groups=5)),
        (TypeError, lambda: qf.gemm(x, w, out=e(24, 72), compute_dtype="f32")),
        (qb._lib.QbError, lambda: qf.gemm(x, wq, out=e(24, 72), compute_dtype="bf16")),
        (ValueError, lambda: qf.ada_rmsnorm(x, row, w, out=e(24, 256))),
        (TypeError, lambda: qf.rmsnorm(wq, out=e(72, 256))),
        (ValueError, lambda: qf.silu(x, out=e(24, 248))),
        (ValueError, lambda: qf.add(x, w, out=e(24, 256))),
        (TypeError, lambda: qf.euler_step(x, y, row, out=e(24, 256))),
        (ValueError, lambda: qf.quantize_e4m3(x, out=e(24, 256))),
        (TypeError, lambda: qf.dequantize_e4m3(x, out=e(24, 256))),
    ]
    first = [c().to_numpy() for c in calls]
    for kind, c in wrong:
        with pytest.raises(kind):
            c()
    monkeypatch.setattr(qf, "_fast", qb._lib._NoFastcall())
    for a, c in zip(first, calls):
        np.testing.assert_array_equal(a, c().to_numpy())
    for kind, c in wrong:
        with pytest.raises(kind):
            c()
    assert f32(first[0], "bf16").any()


@pytest.mark.parametrize("rows", [1, 148, 149])  # up to a row per SM, and more
@pytest.mark.parametrize("D", [8, 2048, 2056, 4104, 8192])  # one, two and four vectors a thread, rows that end inside one
def test_ada_rmsnorm_rows_and_widths(qb, rows, D):
    r = util.rng([98, rows, D])
    X, s, b = bf16_randn(r, (rows, D)), bf16_randn(r, (1, D), 0.1), bf16_randn(r, (1, D), 0.1)
    outq = qb.QuarkTensor.empty(rows, D, dtype="e4m3")
    args = (T(qb, X, "bf16"), T(qb, s, "bf16"), T(qb, b, "bf16"))
    first = qb.qf.ada_rmsnorm(*args, out_q=outq)
    got, want = first.to_numpy(), ops.ada_rmsnorm(X, s, b)
    # (the tolerance of the norm's own test: the sums differ in order only)
    assert np.percentile(util.bf16_ulp_diff(got, want), 99.9) <= 1
    np.testing.assert_array_equal(outq.to_numpy(), codec.f32_to_e4m3(codec.bf16_to_f32(got)))
    # in a chain each call waits for the one before it
    again = qb.qf.ada_rmsnorm(qb.qf.ada_rmsnorm(*args), *args[1:]).to_numpy()
    assert np.percentile(util.bf16_ulp_diff(again, ops.ada_rmsnorm(got, s, b)), 99.9) <= 1


@pytest.mark.parametrize("rows", [1, 148, 149])  # a chained call rehearses with up to a row per SM
@pytest.mark.parametrize("D", [8, 2056, 8192])
def test_ada_rmsnorm_between_other_kernels_gives_the_same_bytes(qb, rows, D):
    r = util.rng([93, rows, D])
    args = T(qb, bf16_randn(r, (rows, D)), "bf16"), T(qb, bf16_randn(r, (1, D), 0.1), "bf16"), T(qb, bf16_randn(r, (1, D), 0.1), "bf16")
    for kw in ({}, dict(activation="silu")):
        want, want_q = qb.qf.ada_rmsnorm(*args, **kw).to_numpy(), qb.QuarkTensor.empty(rows, D, dtype="e4m3")
        qb.qf.ada_rmsnorm(*args, out_q=want_q, only_q=True, **kw)
        # made by Python (an output to be allocated) and in C, behind a kernel that writes its input
        x, q = qb.QuarkTensor.zeros(rows, D, dtype="bf16"), qb.QuarkTensor.empty(rows, D, dtype="e4m3")
        zero = qb.QuarkTensor.zeros(rows, D, dtype="bf16")
        qb.qf.add(args[0], zero, out=x)
        got = qb.qf.ada_rmsnorm(x, *args[1:], chained=True, **kw)
        qb.qf.add(args[0], zero, out=x)
        qb.qf.ada_rmsnorm(x, *args[1:], out_q=q, only_q=True, chained=True, **kw)
        np.testing.assert_array_equal(got.to_numpy(), want)
        np.testing.assert_array_equal(q.to_numpy(), want_q.to_numpy())

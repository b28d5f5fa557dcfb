"""Host logic of the shared scratch buffers of ``qf.*`` (no GPU: the device tensor class is replaced by a stand-in)."""

import ctypes as C

import pytest


class _FakeTensor:
    _next = 0x1000

    def __init__(self, nbytes):
        self.nbytes = nbytes
        self.addr = _FakeTensor._next
        _FakeTensor._next += 0x100000

    @classmethod
    def zeros(cls, n, dtype="e4m3"):
        return cls(int(n))

    def data_ptr(self):
        return self.addr


def test_a_workspace_that_grows_is_retired_not_freed(monkeypatch):
    """A CUDA graph captured while a smaller workspace was current holds that buffer's address; dropping the
    last reference would free it under the graph.  The replaced buffer must stay owned by the module."""
    from quark_b200 import functional as qfm

    monkeypatch.setattr(qfm, "QuarkTensor", _FakeTensor)
    monkeypatch.setattr(qfm, "_WS", None)
    monkeypatch.setattr(qfm, "_ATTN_WS", None)
    monkeypatch.setattr(qfm, "_RETIRED_WS", [])
    first = qfm._workspace(4096)
    assert first.nbytes >= 1 << 20 and qfm._workspace(8192) is first and qfm._workspace(0) is first
    captured_address = first.data_ptr()
    second = qfm._workspace(64 << 20)
    assert second is not first and second.nbytes >= 64 << 20
    assert any(t is first for t in qfm._RETIRED_WS) and first.data_ptr() == captured_address
    a1 = qfm._attn_workspace(1 << 16)
    a2 = qfm._attn_workspace(1 << 24)
    assert a2 is not a1 and any(t is a1 for t in qfm._RETIRED_WS) and qfm._attn_workspace(0) is None


def test_streams_and_graphs_have_workspaces_of_their_own(monkeypatch):
    """Tickets and partial results lie in the workspace, so calls that may overlap must not share one: calls on two streams, and a
    captured graph and anything else."""
    from quark_b200 import functional as qfm
    from quark_b200.runtime import stream

    monkeypatch.setattr(qfm, "QuarkTensor", _FakeTensor)
    for name, value in (("_WS", None), ("_ATTN_WS", None), ("_RETIRED_WS", []), ("_OF_STREAM", type(qfm._OF_STREAM)())):
        monkeypatch.setattr(qfm, name, value)
    monkeypatch.setattr(stream, "_stream", 1)
    both = lambda: (qfm._workspace(4096), qfm._attn_workspace(4096))  # noqa: E731
    first = both()
    stream.set_stream(2)
    second = both()
    assert not {t.data_ptr() for t in first} & {t.data_ptr() for t in second}
    stream.set_stream(1)
    assert both() == first
    stream.set_stream(1)
    assert both() == first and list(qfm._OF_STREAM) == [2]

    graph = stream.Graph(0)
    for f in stream.on_captured:
        f(graph)
    assert graph.scratch == first and not set(both()) & set(first)  # allocated already: the next capture may not

    # bounded: the workspaces of the stream that was left first are taken over once the device is idle
    synced = []
    monkeypatch.setattr(qfm._lib, "load", lambda: type("Lib", (), {"qb_device_sync": staticmethod(lambda: synced.append(1) or 0)}))
    seen = {both()[0]}
    for s in range(10, 60):
        stream.set_stream(s)
        seen.add(both()[0])
    assert synced and len(seen) <= qfm._STREAMS_KEPT + 2 and len(qfm._OF_STREAM) <= qfm._STREAMS_KEPT


def test_counter_and_ticket_areas_do_not_depend_on_the_shape():
    """Calls of different shapes share one workspace, so the area that must stay zero between calls (tile
    counters of the GEMM, tickets of the attention key splits) has to end at the same offset for all of them."""
    from quark_b200 import _lib

    lib = _lib.load()

    def gemm_ws(M, N, K, split_k, a_dtype=1):
        p = _lib.GemmParams(M=M, N=N, K=K, a_dtype=a_dtype, b_dtype=1, c_dtype=0, compute_dtype=1, gate_groups=1, split_k=split_k, tile_n=64,
                            reserved=1)  # fmt: skip
        return int(lib.qb_gemm_workspace_bytes(C.byref(p)))

    counters = 64 << 10
    assert gemm_ws(128, 256, 512, 1) == 0  # e4m3 A, one slice: no scratch memory at all
    assert gemm_ws(128, 256, 512, 1, a_dtype=0) == counters + 128 * 512  # the e4m3 copy of a bf16 A follows the counters
    assert gemm_ws(512, 4096, 768, 3) == counters + 3 * 512 * 4096 * 4  # 256 tiles
    assert gemm_ws(1024, 4096, 768, 3) == counters + 3 * 1024 * 4096 * 4  # 512 tiles: same counter area


def test_attention_asks_only_for_scratch_that_it_uses():
    """Key splits of the kernel's own choice meet inside a cluster: no workspace.  Forced splits and the helpers of a long history use one."""
    from quark_b200 import _lib

    lib = _lib.load()

    def scratch(H, W, Hk, nb=16, splits=0):
        p = _lib.AttnParams(n_kv_heads=Hk, gqa_ratio=2, H_spatial=H, W_spatial=W, num_buckets=nb, pinned_dilation=1, kv_dtype=1, compute_dtype=1,
                            max_segments=3, packed_qkv=1, quilt_factor=1, kv_splits=splits)  # fmt: skip
        return int(lib.qb_owl_attn_scratch_bytes(C.byref(p)))

    per = 66 * 128 * 4
    assert scratch(16, 8, 16) == scratch(32, 16, 2) == scratch(32, 16, 16) == 0
    assert scratch(16, 8, 16, splits=4) == 16384 + 32 * 4 * per
    assert scratch(32, 16, 16, nb=128) == 16384 + 2 * 148 * per


def test_parameter_structs_kept_do_not_loosen_a_check(monkeypatch):
    """A struct is found again by its plain integers alone: a float that equals one of them is refused as it is without the lookup, and
    a struct with addresses in it is not kept."""
    from quark_b200 import _lib
    from quark_b200 import functional as qfm

    monkeypatch.setattr(qfm, "_PARAMS", {})
    sizes = (4, 2, 8, 8, 16, 1, 1, 3, 1, 1, 0)
    kept = qfm._params(_lib.KvParams, *sizes, None, None)
    assert qfm._params(_lib.KvParams, *sizes, None, None) is kept and len(qfm._PARAMS) == 1
    with pytest.raises(TypeError):
        qfm._params(_lib.KvParams, 4, 2.0, *sizes[2:], None, None)
    assert qfm._params(_lib.KvParams, *sizes, 4096, None)[0].k_scale == 4096
    assert qfm._params(_lib.KvParams, True, *sizes[1:], None, None)[0].n_q_heads == 1
    assert len(qfm._PARAMS) == 1

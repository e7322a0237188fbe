"""Sizes at which the selection and the fused preparation change shape: edges of their tiles and groups, the smallest and
largest member of each dispatch, against the oracle or the path that the other tests compare with it."""
import ctypes
import subprocess
import sys
import threading

import pytest
import torch

import sparge_oracle as O

pytestmark = pytest.mark.gpu


def _pooled(BH, nq, nk, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    pq, pk = torch.randn(1, BH, nq, D, generator=g) * 0.7, torch.randn(1, BH, nk, D, generator=g)
    sim_q, sim_k = (torch.rand(1, BH, nq, generator=g) > 0.2), (torch.rand(1, BH, nk, generator=g) > 0.1)
    return pq.to(dtype), pk.to(dtype), sim_q, sim_k


# key blocks around the 64-row score tile, the 256-key group and the 16-byte load; 1 024 and 2 049 with few rows take the
# widest cumsum chunks, 63 with many rows the narrowest
@pytest.mark.parametrize("BH,nq,nk", [(1, 1, 1), (2, 3, 7), (1, 5, 63), (2, 4, 64), (3, 3, 65), (1, 6, 255), (2, 2, 256), (1, 3, 257),
                                      (24, 32, 63), (1, 2, 1024), (1, 1, 2049)])
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.float16, 64)])
@pytest.mark.parametrize("causal", [False, True])
def test_selection_at_tile_edges(BH, nq, nk, dtype, D, causal):
    from spargeattn_b200 import ops
    pq, pk, sim_q, sim_k = _pooled(BH, nq, nk, D, dtype, 100 * nk + nq)
    p = O.pooled_probs(pq, pk, sim_k, causal)
    dev = [t.cuda() for t in (pq, pk, sim_q.to(torch.uint8), sim_k.to(torch.uint8))]
    for topk, cdf in ((0.37, None), (None, 0.9)):
        knob = torch.full((BH,), topk or cdf)
        want = O.select_blocks(p, sim_q, sim_k, knob if topk else None, knob if cdf else None, causal, nk > 64)
        lut, valid, mask = ops.select_blocks(*dev, knob.cuda() if topk else None, knob.cuda() if cdf else None, causal, nk > 64, True)
        assert torch.equal(mask.cpu().bool(), want)
        lut_o, valid_o = O.block_map_to_lut(want)
        assert torch.equal(lut.cpu(), lut_o) and torch.equal(valid.cpu(), valid_o)


@pytest.mark.parametrize("BH,nq,nk", [(40, 119, 238), (37, 128, 31)])
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float16, 128)])
def test_selection_with_two_rows_per_warp(BH, nq, nk, dtype, D):
    """Problems of many rows run two rows per warp; a single head of them runs one."""
    from spargeattn_b200 import ops
    dev = [t.cuda() for t in _pooled(BH, nq, nk, D, dtype, 7)]
    dev[2:] = [t.to(torch.uint8) for t in dev[2:]]
    knob = torch.linspace(0.1, 0.9, BH).cuda()
    for causal in (False, True):
        lut, valid, mask = ops.select_blocks(*dev, knob, None, causal, True, True, best_first=True)
        for h in (0, BH // 2, BH - 1):
            one = ops.select_blocks(*[t[:, h:h + 1].contiguous() for t in dev], knob[h:h + 1], None, causal, True, True, best_first=True)
            for a, b in zip((lut, valid, mask), one):
                assert torch.equal(a[:, h:h + 1], b)


# around the 256-token span, the block sizes inside it and the size from which partial results are combined by a kernel
@pytest.mark.parametrize("N", [128, 129, 255, 256, 257, 511, 2048, 2049, 2300])
@pytest.mark.parametrize("D,dtype,v_dtype", [(64, torch.bfloat16, torch.bfloat16), (128, torch.float16, torch.float16),
                                             (128, torch.bfloat16, torch.float16)])
def test_fused_preparation_equals_the_separate_kernels(N, D, dtype, v_dtype):
    import spargeattn_b200 as S
    from spargeattn_b200 import core, ops
    g = torch.Generator().manual_seed(N + D)
    q, k, v = (torch.randn(2, 3, N, D, generator=g).cuda().to(t) for t in (dtype, dtype, v_dtype))
    k = k + 2
    # token-major V of one dtype with Q: what the fp16-PV path reads through its strides
    v_nhd = v.transpose(1, 2).contiguous().transpose(1, 2)
    calls = [lambda: S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.5, pvthreshd=6.0),
             lambda: S.spas_sage2_attn_meansim_topk_cuda(q, k, v_nhd, topk=0.5, smooth_k=False, is_causal=True),
             lambda: S.spas_sage_attn_meansim_topk_cuda(q, k, v, topk=0.5),
             lambda: S.spas_sage_attn_meansim_topk_cuda(q, k, v_nhd, topk=0.5, is_causal=True),
             lambda: S.spas_sage_attn_meansim_topk_cuda(q, k, v[:, :1].expand(2, 3, N, D), topk=0.5)]
    one = [f() for f in calls]
    limit = core.SINGLE_CALL_MAX_ROWS
    try:
        core.SINGLE_CALL_MAX_ROWS = 0
        sep = [f() for f in calls]
    finally:
        core.SINGLE_CALL_MAX_ROWS = limit
    for a, b in zip(one, sep):
        assert torch.equal(a, b)
    # block mask: composed from the separate entries
    mask = torch.rand(2, 3, (N + 127) // 128, (N + 63) // 64, generator=g) < 0.6
    for m in (mask.cuda(), mask.to(torch.int64).cuda()):
        o = S.block_sparse_sage2_attn_cuda(q, k, v, mask_id=m)
        q8, qs, k8, ks = core.get_vanilla_qk_quant(q, k, ops.k_mean(k))
        lut, valid = ops.mask_to_lut(m)
        v8, vs = ops.quant_v(v)
        assert torch.equal(o, ops.attn_fwd(q8, k8, v8, lut, valid, None, qs, ks, vs, D ** -0.5, False, dtype))
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 6e4])
def test_selection_of_rows_without_defined_probabilities(dtype, causal, value):
    """NaN, infinite and (6e4 in fp16) overflowing scores: the first blocks of the row are selected, not all of them."""
    from spargeattn_b200 import ops
    pq, pk, sim_q, sim_k = _pooled(2, 40, 70, 64, dtype, 3)
    sim_q[:] = True
    pq[0, 0, 30, 5] = value
    pk[0, 1, 9] = value
    dev = [t.cuda() for t in (pq, pk, sim_q.to(torch.uint8), sim_k.to(torch.uint8))]
    p = O.pooled_probs(pq, pk, sim_k, causal)
    for topk, cdf in ((0.1, None), (None, 0.7)):
        knob = torch.full((2,), topk or cdf)
        want = O.select_blocks(p, sim_q, sim_k, knob if topk else None, knob if cdf else None, causal, False)
        lut, valid, mask = ops.select_blocks(*dev, knob.cuda() if topk else None, knob.cuda() if cdf else None, causal, False, True)
        assert torch.equal(mask.cpu().bool(), want)
        lut_o, valid_o = O.block_map_to_lut(want)
        assert torch.equal(lut.cpu(), lut_o) and torch.equal(valid.cpu(), valid_o)


def _in_new_process(call):
    """Kernel attributes outlive a call: what a launch needs shows only where no larger one came before it."""
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:0] = {sys.path!r}; import test_gpu_edges as t; t.{call}"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


def _check_cdf_selection(BH, nq, nk):
    from spargeattn_b200 import ops
    pq, pk, sim_q, sim_k = _pooled(BH, nq, nk, 64, torch.float16, nk)
    knob = torch.full((BH,), 0.9)
    want = O.select_blocks(O.pooled_probs(pq, pk, sim_k, False), sim_q, sim_k, None, knob, False, False)
    dev = [t.cuda() for t in (pq, pk, sim_q.to(torch.uint8), sim_k.to(torch.uint8))]
    assert torch.equal(ops.select_blocks(*dev, None, knob.cuda(), False, False, True)[2].cpu().bool(), want)


# four rows take exactly 48 KB of dynamic shared memory from 1 281 to 1 408 blocks (with the scan's chunk, which follows the
# number of rows), the first size above it is 1 409
@pytest.mark.parametrize("BH,nq,nk", [(2, 64, 1281), (2, 64, 1408), (2, 64, 1409), (1, 600, 1345), (3, 700, 1377)])
def test_cdf_selection_where_dynamic_shared_memory_reaches_48_kb(BH, nq, nk):
    _in_new_process(f"_check_cdf_selection({BH}, {nq}, {nk})")


def _check_mask_to_lut(nk):
    from spargeattn_b200 import ops
    m = torch.rand(1, 1, 2, nk, generator=torch.Generator().manual_seed(nk)) < 0.5
    lut, valid = ops.mask_to_lut(m.cuda())
    lut_o, valid_o = O.block_map_to_lut(m)
    assert torch.equal(lut.cpu(), lut_o) and torch.equal(valid.cpu(), valid_o)


# around the 48 KB that a launch may ask for without the attribute, and the longest row
@pytest.mark.parametrize("nk", [12280, 12281, 12288, 12289, 51200])
def test_block_mask_rows_where_dynamic_shared_memory_reaches_48_kb(nk):
    _in_new_process(f"_check_mask_to_lut({nk})")


def _check_capture_with_a_known_knob():
    import spargeattn_b200 as S
    g = torch.Generator().manual_seed(5)
    q, k, v = (torch.randn(1, 2, 512, 64, generator=g).bfloat16().cuda() for _ in range(3))
    S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.5)
    want, _ = S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.4375, return_sparsity=True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        o = S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.4375)
    graph.replay()
    assert torch.equal(o, want)


def test_a_knob_that_one_entry_has_seen_can_be_captured_by_another():
    _in_new_process("_check_capture_with_a_known_knob()")


def test_a_knob_beyond_fp32_is_refused():
    import spargeattn_b200 as S
    q = torch.randn(1, 2, 256, 64).bfloat16().cuda()
    for kw in ({"topk": 1e300}, {"topk": 1e300, "return_sparsity": True}, {"pvthreshd": -1e300}):
        with pytest.raises(RuntimeError):
            S.spas_sage2_attn_meansim_topk_cuda(q, q, q, **kw)


def test_a_share_without_query_blocks_leaves_the_output_alone():
    """Every CTA of the attention kernel leaves at once; what follows on the stream reuses the call's workspace."""
    from spargeattn_b200.sharding import attention_units
    import spargeattn_b200 as S
    g = torch.Generator().manual_seed(6)
    q, k, v = (torch.randn(1, 2, 2304, 128, generator=g).bfloat16().cuda() for _ in range(3))
    want = S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.5)
    none = torch.zeros(1, 2, 2, dtype=torch.int32, device="cuda")
    for _ in range(20):
        attention_units(q, k, v, none, 1, topk=0.5)
        assert torch.equal(S.spas_sage2_attn_meansim_topk_cuda(q, k, v, topk=0.5), want)


def test_a_refused_launch_leaves_no_error_behind():
    """Launches into a capture that has been invalidated are refused by the runtime: the call says so, and the thread's last
    error, which the next check of anybody's launch would report, stays clear."""
    from spargeattn_b200 import _cabi, ops
    rt = ctypes.CDLL("libcudart.so.12")
    mask = torch.ones(1, 1, 2, 4, dtype=torch.uint8, device="cuda")
    lut, valid = torch.empty(1, 1, 2, 4, dtype=torch.int32, device="cuda"), torch.empty(1, 1, 2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0                     # relaxed: nothing else of the process is held up
    assert rt.cudaStreamSynchronize(stream) != 0                         # not allowed in a capture: invalidates it
    rt.cudaGetLastError()
    status = _cabi.lib.sparge_mask_to_lut(mask.data_ptr(), 1, lut.data_ptr(), valid.data_ptr(), 1, 1, 2, 4, stream)
    left = rt.cudaGetLastError()
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    rt.cudaGetLastError()
    assert rt.cudaStreamDestroy(stream) == 0
    assert status == _cabi.ERR_CUDA and left == 0
    assert ops.mask_to_lut(mask)[1].tolist() == [[[4, 4]]]


def test_rows_of_different_lengths_from_several_threads():
    """The kernels' shared-memory attribute is common to all threads: a short row must not take a long one's away."""
    from spargeattn_b200 import ops
    problems = []

    def run(nk):
        try:
            dev = [t.cuda() for t in _pooled(1, 4, nk, 128, torch.bfloat16, nk)]
            dev[2:] = [t.to(torch.uint8) for t in dev[2:]]
            knob, mask = torch.full((1,), 0.5).cuda(), torch.ones(1, 1, 1, nk + 12000, dtype=torch.uint8, device="cuda")
            for _ in range(2000):
                ops.select_blocks(*dev, knob, None, False, False)
                ops.mask_to_lut(mask)
        except Exception as e:
            problems.append(e)

    threads = [threading.Thread(target=run, args=(nk,)) for nk in (4000, 4600, 12000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not problems


@pytest.mark.parametrize("ranges", [[0, 1, 0, 1], "0101", torch.zeros(1, 2, 2), torch.zeros(1, 2, 2, dtype=torch.int32), None])
def test_row_ranges_that_are_no_device_tensor(ranges):
    """What the binding cannot take it leaves to the general path, which complains; without ranges it takes the call."""
    from spargeattn_b200 import core
    q = torch.randn(1, 2, 256, 64).bfloat16().cuda()
    args = (False, None, True, -0.1, None, 0.5, 50, False, "HND", False, False)
    r = core._binding.forward(q, q, q, None, -0.1, None, 0.5, 50, None, False, False, False, True, False, "HND", ranges, 1, False)
    if ranges is None:
        assert torch.equal(r, core._meansim_attention(q, q, q, *args))
    else:
        assert r is None
        with pytest.raises((AttributeError, AssertionError, RuntimeError)):
            core._meansim_attention(q, q, q, *args, q_block_ranges=ranges, q_blocks_max=1)


def test_block_mask_entry_refuses_other_head_sizes_with_a_value_error():
    import spargeattn_b200 as S
    q, ok = (torch.randn(1, 2, 256, d).bfloat16().cuda() for d in (96, 64))
    mask = torch.ones(1, 2, 2, 4, dtype=torch.bool, device="cuda")
    for kw in ({"mask_id": mask}, {"mask_id": mask, "smooth_k": False}, {"mask_id": None}, {"mask_id": mask, "return_sparsity": True}):
        with pytest.raises(ValueError):
            S.block_sparse_sage2_attn_cuda(q, q, q, **kw)
    for mask_id in (None, mask[0], mask.transpose(2, 3)):
        with pytest.raises(AssertionError):
            S.block_sparse_sage2_attn_cuda(ok, ok, ok, mask_id=mask_id)


@pytest.mark.parametrize("kw", [dict(topk=0.4), dict(topk=0.4, pvthreshd=4.0, is_causal=True), dict(cdfthreshd=0.9, simthreshd1=0.3),
                                dict(cdfthreshd=0.8, pvthreshd=4.0, attention_sink=True, smooth_k=False)])
@pytest.mark.parametrize("N,D,dtype,v_dtype", [(1000, 64, torch.bfloat16, torch.float16), (2048, 128, torch.float16, torch.float16),
                                               (2500, 128, torch.bfloat16, torch.bfloat16)])
def test_c_entry_of_the_whole_path(kw, N, D, dtype, v_dtype):
    """The C signature: its strides, the parts at the reported offsets, a workspace of exactly the reported size."""
    import spargeattn_b200 as S
    from spargeattn_b200 import _cabi, core, ops
    B, H = 2, 3
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(B, N, H, D, generator=g).to(t).cuda().transpose(1, 2) for t in (dtype, dtype, v_dtype))   # token-major
    causal, sink, smooth = kw.get("is_causal", False), kw.get("attention_sink", False), kw.get("smooth_k", True)
    fn = S.spas_sage2_attn_meansim_topk_cuda if "topk" in kw else S.spas_sage2_attn_meansim_cuda
    want = fn(q, k, v, **{"simthreshd1": -0.1, **kw})
    vec = lambda name, default=None: None if kw.get(name, default) is None else torch.full((H,), kw.get(name, default), device="cuda")
    thr, cdf, topk, pv = vec("simthreshd1", -0.1), vec("cdfthreshd"), vec("topk"), vec("pvthreshd")
    o, ws, at = ops.meansim_forward(q, k, v, torch.empty(B, H, N, D, dtype=dtype, device="cuda"), thr, cdf, topk, pv, D ** -0.5, causal,
                                    False, sink, smooth)
    assert torch.equal(o, want)
    # the parts, against the separate entries
    km = ops.k_mean(k) if smooth else None
    pq, sq, q8, qs = ops.pool_sim_quant(q, None, 128, thr)
    pk, sk, k8, ks = ops.pool_sim_quant(k, km, 64, thr)
    lut, valid, _ = ops.select_blocks(pq, pk, sq, sk, topk, cdf, causal, sink, best_first=pv is None)
    v8, vs = ops.quant_v(v)
    parts = dict(pq=pq, pk=pk, sim_q=sq, sim_k=sk, q_int8=q8, k_int8=k8, q_scale=qs, k_scale=ks, lut=lut, valid=valid, v8=v8, v_scale=vs)
    if smooth:
        parts["km"] = km
    assert set(ops.WS_PARTS) == set(parts) | {"scratch", "km"}
    for name, t in parts.items():
        assert torch.equal(ws[at[name]:at[name] + t.numel() * t.element_size()], t.contiguous().view(-1).view(torch.uint8)), name
    # one byte short is refused, exactly enough does not touch what lies behind
    nbytes = int(_cabi.lib.sparge_forward_workspace_bytes(B, H, N, D))
    guarded, out = torch.full((nbytes + 4096,), 0x5a, dtype=torch.uint8, device="cuda"), torch.empty_like(q)
    st3 = lambda t: (ctypes.c_longlong * 3)(*t.stride()[:3])
    ptr = lambda t: None if t is None else t.data_ptr()
    call = lambda n: _cabi.lib.sparge_meansim_forward(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), ptr(thr), ptr(cdf), ptr(topk), ptr(pv), guarded.data_ptr(), n, None, B, H,
        N, D, ops._dt(q), ops._dt(v), int(causal), 0, int(sink), int(smooth), D ** -0.5, st3(q), st3(k), st3(v), st3(out), None)
    torch.cuda.synchronize()
    assert call(nbytes - 1) == _cabi.ERR_INVALID_ARG
    assert call(nbytes) == _cabi.OK
    torch.cuda.synchronize()
    assert torch.equal(out, want) and bool((guarded[nbytes:] == 0x5a).all())
    ops.check_device_status()


def _rows_of_many_lengths(B, H, N, D, dtype):
    """q, k, v whose query blocks are alike in themselves and look at anything from a few key blocks to nearly all."""
    g = torch.Generator("cuda").manual_seed(N)
    per_block = lambda size: torch.randn(B, H, (N + size - 1) // size, D, generator=g, device="cuda").repeat_interleave(size, 2)[:, :, :N]
    noise = lambda: 0.3 * torch.randn(B, H, N, D, generator=g, device="cuda")
    sharp = (4 * torch.rand(B, H, (N + 127) // 128, 1, generator=g, device="cuda")).repeat_interleave(128, 2)[:, :, :N]
    return (sharp * per_block(128) + noise()).to(dtype), (per_block(64) + noise()).to(dtype), noise().to(dtype)


@pytest.mark.parametrize("kw", [dict(cdfthreshd=0.8, simthreshd1=-0.1), dict(topk=0.3, is_causal=True), dict(cdfthreshd=0.7, is_causal=True, pvthreshd=4.0),
                                dict(cdfthreshd=0.8, simthreshd1=-0.1, fp16_pv=True), dict(topk=0.3, is_causal=True, fp16_pv=True)])
@pytest.mark.parametrize("B,H,N,D,layout", [(1, 148, 256, 64, "HND"), (1, 297, 128, 64, "HND"), (1, 5, 7700, 128, "HND"), (1, 41, 4996, 128, "HND"),
                                            (1, 41, 5200, 128, "HND"), (2, 4, 5190, 64, "NHD"), (2, 25, 10300, 64, "HND"), (3, 2, 6700, 128, "NHD")])
def test_longest_rows_first(kw, B, H, N, D, layout):
    """Rows that differ in length are computed in another order, sorted by their counts in cdf calls of more than 296 rows of
    more than 80 blocks, by position in the other causal ones: one group of heads and several, one batch and several, both
    kinds of V. Every row has to come out, with the bytes of the separate entries, which compute them in their own order."""
    import spargeattn_b200 as S
    from spargeattn_b200 import core, ops
    kw = dict(kw, tensor_layout=layout)
    fp16_pv = kw.pop("fp16_pv", False)
    q, k, v = _rows_of_many_lengths(B, H, N, D, torch.float16 if fp16_pv else torch.bfloat16)
    if layout == "NHD":
        q, k, v = (x.transpose(1, 2).contiguous() for x in (q, k, v))
    sage = "sage" if fp16_pv else "sage2"
    fn = getattr(S, f"spas_{sage}_attn_meansim_topk_cuda" if "topk" in kw else f"spas_{sage}_attn_meansim_cuda")
    del_me = torch.full_like(q, float("nan"))              # what the output's memory holds: a row left out shows
    del del_me
    one = fn(q, k, v, **kw)
    single = core.SINGLE_CALL_MAX_ROWS
    try:
        core.SINGLE_CALL_MAX_ROWS = 0
        separate = fn(q, k, v, **kw)
    finally:
        core.SINGLE_CALL_MAX_ROWS = single
    ops.check_device_status()
    assert torch.equal(one, separate)


@pytest.mark.parametrize("B,H,N,D,ordered", [(1, 6, 6400, 128, True), (2, 25, 5300, 128, True), (1, 21, 33000, 64, True), (3, 9, 33000, 128, True),
                                             (1, 8, 5120, 64, False), (1, 8, 5121, 64, True),       # 80, 81 blocks
                                             (1, 4, 9472, 64, False), (1, 3, 12672, 64, True)])     # 296, 297 rows
def test_order_of_the_rows(B, H, N, D, ordered):
    """The sorted order that a cdf call of more than 296 rows of more than 80 blocks leaves in its workspace: every row once, in
    even groups of heads (as many heads as have their K and V in some tens of MB; a short last group starts its longest rows
    late), longest first in each group. A bucket is 1/255 of a row."""
    from spargeattn_b200 import ops
    q, k, v = _rows_of_many_lengths(B, H, N, D, torch.bfloat16)
    vec = lambda x: torch.full((H,), x, device="cuda")
    _, ws, at = ops.meansim_forward(q, k, v, torch.empty_like(q), vec(-0.1), vec(0.8), None, None, D ** -0.5, False, False, False, True)
    ops.check_device_status()
    nq, nk = (N + 127) // 128, (N + 63) // 64
    part = lambda name: ws[at[name]:at[name] + B * H * nq * 4].view(torch.int32).cpu().long()
    rows, valid = part("scratch"), part("valid")
    assert torch.equal(rows.sort().values, torch.arange(B * H * nq)) == ordered
    if not ordered:
        return
    assert valid.max() - valid.min() > nk // 4                                     # the order is put to a test
    ends = (rows.cummax(0).values == torch.arange(B * H * nq)).nonzero().flatten() + 1   # the first n rows are 0 .. n - 1
    ends = [0] + [int(e) for e in ends if e % nq == 0]
    heads = [(b - a) // nq for a, b in zip(ends, ends[1:])]
    assert sum(heads) == B * H and max(heads) - min(heads) <= 1 and max(heads) > 1, heads
    bucket = 255 - valid[rows] * 255 // nk
    for a, b in zip(ends, ends[1:]):
        assert bool((bucket[a:b].diff() >= 0).all())


def test_ranges_without_a_largest_count_are_an_assertion():
    from spargeattn_b200.sharding import attention_units
    q = torch.randn(1, 2, 256, 64).bfloat16().cuda()
    for largest in (None, 0, -1):                          # None: read back from the ranges, which are empty
        with pytest.raises(AssertionError):
            attention_units(q, q, q, torch.zeros(1, 2, 2, dtype=torch.int32), largest, topk=0.5)


def test_native_calls_on_several_streams_and_threads():
    """Each call takes its workspace and output on the stream it runs on; scalar knobs are shared."""
    import spargeattn_b200 as S
    g = torch.Generator().manual_seed(8)
    x = [[torch.randn(1, 2, n, 128, generator=g).bfloat16().cuda() for _ in range(3)] for n in (700, 1500, 2600, 4000)]
    call = lambda i, j: S.spas_sage2_attn_meansim_topk_cuda(*x[i], topk=0.3 + 0.01 * j, is_causal=j % 2 == 1)
    want = [[call(i, j) for j in range(4)] for i in range(4)]
    torch.cuda.synchronize()
    got = [[] for _ in range(4)]

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = [call((i + r) % 4, r % 4) for r in range(40)]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        assert len(got[i]) == 40 and all(torch.equal(o, want[(i + r) % 4][r % 4]) for r, o in enumerate(got[i]))

"""Single-GPU tests: every kernel at world_size 1 against plain PyTorch fp32/fp64 math."""
import pytest
import torch

from amd_distributed_2025_b200 import contract, oracle

pytestmark = pytest.mark.gpu


def _ext():
    from amd_distributed_2025_b200.ops import _ext

    return _ext.load()


# The planners of the one-rank GEMM and of the fp8 GEMM are functions of the problem's size, the number of SMs and how many
# clusters of 2, 3 .. 16 CTAs fit on the device at once.  Sizes that are to reach a certain path are chosen for this part.
_PART = (148, (74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7))


def _check_plan(got, want):
    part = (torch.cuda.get_device_properties(0).multi_processor_count, tuple(_ext().gemm_cluster_capacity(i) for i in range(2, 17)))
    if part != _PART:
        pytest.skip(f"right, and planned here as {got}: this part has {part}, the size is chosen for {_PART}")
    assert got == want


def test_extension_is_loaded_from_tree():
    mod = _ext()
    assert mod.__file__.endswith("_C/b200_ext.so")


def test_bounded_wait_times_out_and_context_survives():
    from amd_distributed_2025_b200.parallel.symm_mem import SlabLayout, SymmetricWorkspace
    from amd_distributed_2025_b200.utils.status import StatusError

    ext = _ext()
    ws = SymmetricWorkspace(SlabLayout(ext.HEAP_HEADER_BYTES), rank=0, world_size=1, wait_limit_ms=5)
    ws.check(sync=True)
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    ws.heap.wait_selftest(3, 12345, 5_000_000)  # a flag nothing sets, 5 ms limit
    stop.record()
    torch.cuda.synchronize()
    assert 4.0 < start.elapsed_time(stop) < 500.0
    with pytest.raises(StatusError) as err:
        ws.check(sync=True)
    assert err.value.code == "timeout" and err.value.phase == "selftest" and err.value.status["peer"] == 3
    assert ws.status()["code"] == 1  # host mirror, no synchronisation needed
    ws.reset_status()
    ws.check(sync=True)
    # the context is still usable
    assert float(torch.ones(4, device="cuda").sum()) == 4.0
    ws.barrier()
    torch.cuda.synchronize()
    ws.check(sync=True)
    ws.close()


@pytest.mark.parametrize("mode", ["dedup", "direct"])
@pytest.mark.parametrize(
    "E,k,H,T,dtype,fixed",
    [
        (8, 2, 6144, 4, torch.float16, None),
        (64, 6, 2048, 8, torch.float16, None),
        (128, 4, 2880, 32, torch.float16, None),
        (256, 8, 7168, 128, torch.bfloat16, 128),
        (16, 2, 256, 32, torch.float32, 32),
        (64, 6, 1024, 1024, torch.bfloat16, 1024),  # > 4096 entries: the grid-barrier kernels
        (256, 8, 512, 600, torch.float16, 600),
        (8, 2, 250, 5, torch.float16, 5),  # row size not a multiple of 16 bytes: scalar paths
    ],
)
def test_moe_world1_matches_oracle(E, k, H, T, dtype, fixed, mode):
    from amd_distributed_2025_b200.models import moe_all2all

    for it in range(3):  # new inputs (and token counts) every call: nothing of the previous call may survive
        n_tok = None if fixed is None else max(fixed - 3 * it, 1)
        cfg, data, rank, ws = contract.make_moe_inputs(E, k, H, T, 7 + it, 0, 1, device="cuda", dtype=dtype,
                                                       fixed_num_tokens=n_tok, routing="zipf" if T >= 600 else "uniform",
                                                       weights="softmax")
        layer = moe_all2all.get_layer(cfg, 0, 1, mode=mode)
        if it == 1:
            got = layer.dispatch(data.x, data.indices)
            torch.cuda.synchronize()
            layer.check()
            ok, msg = oracle.compare_dispatch_layout(got, oracle.moe_dispatch_oracle(cfg, [data], 0))
            assert ok, msg
            layer.expert_scale(1.0)
            y = torch.empty(data.num_tokens, H, dtype=dtype, device="cuda")
            layer.combine(y, data.weights, got[2], layer.expert_y, got[0], data.num_tokens)
        else:
            y = moe_all2all.custom_kernel((cfg, data, 0, 1), mode=mode)
        torch.cuda.synchronize()
        layer.check()
        ok, msg = oracle.check_moe_output(y, oracle.moe_expected_output(cfg, data, 1))
        assert ok, (it, msg)
        assert oracle.relative_error(y, oracle.moe_expected_output(cfg, data, 1, acc_dtype=torch.float64)) < 5e-3


@pytest.mark.parametrize(
    "E,k,H,T,M,dtype",
    [
        (8, 1, 64, 1, 3, torch.float16),  # one entry, one piece
        (5, 5, 520, 7, 7, torch.bfloat16),  # every expert gets every token; last piece of a row is short
        (64, 6, 1000, 395, 400, torch.float32),  # pieces shared between CTAs, just above 16 warps per SM
        (1030, 3, 24, 1366, 1366, torch.float16),  # more experts than the replicated counts take, rows of 3 vectors
        (16, 8, 256, 4096, 4096, torch.bfloat16),  # the most entries the single launch takes ...
        (16, 8, 256, 4097, 4097, torch.bfloat16),  # ... and one token more
    ],
)
def test_moe_one_rank_kernels_at_the_edges_of_their_ranges(E, k, H, T, M, dtype):
    from amd_distributed_2025_b200.models import moe_all2all

    cfg, data, _, _ = contract.make_moe_inputs(E, k, H, M, 5, 0, 1, device="cuda", dtype=dtype, fixed_num_tokens=T,
                                               routing="zipf", weights="rand")
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
    for scale in (1.0, 3.0):  # the second forward must not see anything of the first
        y = layer.forward(data.x, data.indices, data.weights, scale)
        want = (data.x * scale).double() * data.weights.double().sum(1, keepdim=True)
        assert oracle.relative_error(y, want) < 5e-3
    counts, ex, meta = layer.dispatch(data.x, data.indices)
    ids = data.indices.long().flatten()
    order = torch.sort(ids, stable=True).indices  # entries by expert, (token, k) order inside an expert
    assert torch.equal(counts.long(), torch.bincount(ids, minlength=E))
    slot = torch.arange(T * k, device="cuda") - (torch.cumsum(counts.long(), 0) - counts.long())[ids[order]]
    assert torch.equal(ex[ids[order], slot], data.x[order // k])
    got = meta[ids[order], slot].long()
    assert torch.equal(got, torch.stack([ids[order], 0 * order, order // k, order % k, 0 * order], dim=1))
    ey = torch.randn(ex.shape, device="cuda").to(dtype)
    out = torch.empty(T, H, dtype=dtype, device="cuda")
    layer.combine(out, data.weights, meta, ey, counts, T)
    rows = torch.empty(T * k, H, dtype=torch.float64, device="cuda")
    rows[order] = ey[ids[order], slot].double()
    want = (rows.view(T, k, H) * data.weights.double()[:, :, None]).sum(1)
    assert oracle.relative_error(out, want) < 5e-3
    layer.check()
    layer.close()


@pytest.mark.parametrize(
    "E,k,H,T,dtype",
    [
        (31, 3, 4096, 259, torch.bfloat16),  # forward: 14 pieces per SM, eight warps ...
        (31, 3, 4096, 260, torch.bfloat16),  # ... one piece more, ten
        (40, 5, 4096, 370, torch.bfloat16),  # 20 pieces per SM, ten warps ...
        (40, 5, 4096, 371, torch.bfloat16),  # ... one more, sixteen, and shorter runs for later CTAs
        (40, 2, 4096, 371, torch.bfloat16),  # ... and equal ones with two entries a token
        (9, 3, 512, 3000, torch.float16),  # 20 pieces and a bit per SM, runs of 22 down to 18
        (7, 6, 256, 1024, torch.float16),  # plain dispatch: the most entries that eight warps per CTA take ...
        (7, 6, 256, 1025, torch.float16),  # ... and sixteen; more own entries than one warp ranks at a time
        (130, 5, 1030, 3301, torch.bfloat16),  # rows that are no whole vectors, 16505 entries, own ones not a multiple of 4
        (3, 15, 512, 2184, torch.float32),  # experts that appear several times in a token, nearly 32768 entries
    ],
)
def test_moe_one_rank_shares_of_the_ctas(E, k, H, T, dtype):
    """Where the launcher deals the work out differently, with ids on any address: rows, metadata and counts exactly."""
    from amd_distributed_2025_b200.models import moe_all2all

    cfg = contract.MoEConfig(E, k, H, T * (k if k > E else 1), dtype, dtype)
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=gen).to(dtype)
    w = torch.rand(T, k, device="cuda", generator=gen)
    if k > E:
        ids = torch.randint(0, E, (T, k), device="cuda", generator=gen)
    else:
        ids = torch.rand(T, E, device="cuda", generator=gen).pow(3).argsort(1)[:, :k]
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
    for shift in (0, 1):  # (ids on a 16-byte boundary, and off it)
        idx = torch.empty(T * k + 4, dtype=torch.int32, device="cuda")[shift : shift + T * k].view(T, k).copy_(ids)
        for fused in (True, False):
            layer.expert_x.zero_()  # (what the call before this one left there is not what this one has to write)
            layer.expert_meta.fill_(-1)
            layer.expert_num_tokens.fill_(-1)
            if fused:
                y = layer.forward(x, idx, w, 2.0)
                layer.check()
                assert oracle.relative_error(y, (x * 2.0).double() * w.double().sum(1, keepdim=True)) < 5e-3
            else:
                layer.dispatch(x, idx)
            counts, ex, meta = layer.expert_num_tokens, layer.expert_x, layer.expert_meta
            flat = ids.flatten()
            order = torch.sort(flat, stable=True).indices
            assert torch.equal(counts.long(), torch.bincount(flat, minlength=E))
            slot = torch.arange(T * k, device="cuda") - (torch.cumsum(counts.long(), 0) - counts.long())[flat[order]]
            assert torch.equal(ex[flat[order], slot], x[order // k])
            want = torch.stack([flat[order], 0 * order, order // k, order % k, 0 * order], dim=1)
            assert torch.equal(meta[flat[order], slot].long(), want)
    bad = idx.clone()
    bad[T - 2, k - 1] = E  # known to the last CTAs only as one of their own
    y = layer.forward(x, bad, w, 1.0)
    with pytest.raises(Exception, match="bad_index"):
        layer.check()
    keep = torch.arange(T, device="cuda") != T - 2
    assert oracle.relative_error(y[keep], (x.double() * w.double().sum(1, keepdim=True))[keep]) < 5e-3
    layer.ws.reset_status()
    layer.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 7, 8, 9, 13, 15])
@pytest.mark.parametrize("H,dtype", [(520, torch.bfloat16), (1000, torch.float32), (130, torch.float16)])
def test_moe_one_rank_combine_rounds(k, H, dtype):
    """Every number of rows that combine gathers at a time, and what is left of the last round; pieces that end short, and
    rows that are no whole vectors."""
    _combine_against_fp64(67, 16, k, H, dtype)


@pytest.mark.parametrize("T,k,H", [
    (1183, 3, 4096), (1184, 3, 4096),  # up to three rows: pieces of 1 KiB, and of 2 KiB where each of 4736 warps has one
    (1169, 2, 4152),  # ... the last one 104 bytes long
    (1035, 4, 4096), (1036, 4, 4096),  # more: up to four at a time, and two from 8288 pieces of 1 KiB on
    (1036, 7, 4088), (2072, 13, 2048),  # a last piece that ends short; an odd number of rows
])
def test_moe_one_rank_combine_many_tokens(T, k, H):
    """Where every warp of combine has one piece of a row and more."""
    _combine_against_fp64(T, k + 1, k, H, torch.bfloat16)


def _combine_against_fp64(T, E, k, H, dtype):
    """fp32 sums of k products, rounded once."""
    from amd_distributed_2025_b200.models import moe_all2all

    cfg = contract.MoEConfig(E, k, H, T, dtype, dtype)
    gen = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(T, H, device="cuda", generator=gen).to(dtype)
    w = torch.rand(T, k, device="cuda", generator=gen)
    ids = torch.rand(T, E, device="cuda", generator=gen).argsort(1)[:, :k].int().contiguous()
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
    counts, ex, meta = layer.dispatch(x, ids)
    ey = torch.randn(ex.shape, device="cuda", generator=gen).to(dtype)
    out = layer.combine(torch.empty(T, H, dtype=dtype, device="cuda"), w, meta, ey, counts, T)
    rows = torch.empty(T * k, H, dtype=torch.float64, device="cuda")
    m = meta.long()
    for e in range(E):
        n = int(counts[e])
        rows[m[e, :n, 2] * k + m[e, :n, 3]] = ey[e, :n].double()
    want = (rows.view(T, k, H) * w.double()[:, :, None]).sum(1)
    layer.check()
    eps = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11, torch.float32: 2.0**-23 * (k + 1)}[dtype]
    assert oracle.relative_error(out, want) < eps
    layer.close()


def test_moe_whole_calls_and_the_general_way_agree():
    """custom_kernel, dispatch and combine through the engine's own calls: the layer of each configuration, token counts
    known to what follows, nothing kept of the arguments, wrong ones refused."""
    import sys

    from amd_distributed_2025_b200.models import moe_all2all

    inputs = [contract.make_moe_inputs(E, k, H, 24, 5 + H, 0, 1, device="cuda", dtype=dtype, fixed_num_tokens=T, weights="softmax")
              for E, k, H, T, dtype in ((16, 2, 256, 24, torch.float16), (16, 2, 256, 24, torch.float32), (8, 3, 264, 7, torch.float16))]
    want = [oracle.moe_expected_output(cfg, data, 1) for cfg, data, _, _ in inputs]
    held = None
    for _ in range(3):
        for item, w in zip(inputs, want):  # each its own layer, also right after another's call
            y = moe_all2all.custom_kernel(item)
            assert oracle.check_moe_output(y, w)[0]
        del y, item, w
        if held is None:  # (the layers, made by the first round, hold their configurations)
            held = [sys.getrefcount(v) for cfg, d, _, _ in inputs for v in (cfg, d, d.x, d.indices, d.weights)]
    assert held == [sys.getrefcount(v) for cfg, d, _, _ in inputs for v in (cfg, d, d.x, d.indices, d.weights)]
    cfg, data, _, _ = inputs[2]
    layer = moe_all2all.get_layer(cfg, 0, 1)
    counts, ex, meta = layer.dispatch(data.x, data.indices)
    wide = torch.empty(7, 2 * 264, dtype=torch.float16, device="cuda")[:, :264]  # rows apart: the general way
    with pytest.raises(ValueError):
        layer.combine(wide, data.weights, meta, ex, counts, 6)
    layer.combine(wide, data.weights, meta, ex, counts)
    assert oracle.check_moe_output(wide.contiguous(), want[2])[0]
    for bad in ((data.x,), (data.x, None), (data.x, 3)):
        with pytest.raises(TypeError):
            layer.engine.try_dispatch(*bad)
    moe_all2all.release_layers()  # the layers are gone: new ones
    assert oracle.check_moe_output(moe_all2all.custom_kernel(inputs[0]), want[0])[0]


@pytest.mark.parametrize("mode", ["dedup", "direct"])
def test_moe_combine_takes_the_dispatched_token_count_or_none(mode):
    """Every number but that of the dispatch is refused, negative ones too; whatever int() takes is taken."""
    import numpy

    from amd_distributed_2025_b200.models import moe_all2all

    cfg, data, _, _ = contract.make_moe_inputs(8, 2, 64, 9, 3, 0, 1, device="cuda", dtype=torch.float16, fixed_num_tokens=5)
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode=mode)
    counts, ex, meta = layer.dispatch(data.x, data.indices)
    ey = ex.clone()
    want = oracle.moe_expected_output(cfg, data, 1)  # (one rank scales by 1 + 0)
    for bad in (-1, -5, 0, 4, 6, 2**70, -(2**70)):
        with pytest.raises(ValueError, match="num_tokens"):
            layer.combine(torch.empty(5, 64, dtype=torch.float16, device="cuda"), data.weights, meta, ey, counts, bad)
    for good in (None, 5, 5.0, numpy.int64(5), torch.tensor(5)):
        out = torch.empty(5, 64, dtype=torch.float16, device="cuda")
        layer.combine(out, data.weights, meta, ey, counts, good)
        assert oracle.check_moe_output(out, want)[0]
    layer.check()
    layer.close()


def test_moe_dedup_fp32_partial_rows_and_phase_stamps():
    from amd_distributed_2025_b200.models import moe_all2all

    cfg, data, _, _ = contract.make_moe_inputs(32, 4, 1024, 96, 11, 0, 1, device="cuda", dtype=torch.bfloat16,
                                               fixed_num_tokens=96, weights="softmax")
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup", partial_dtype=torch.float32)
    layer.enable_trace()
    y = layer.forward(data.x, data.indices, data.weights, 1.0)
    torch.cuda.synchronize()
    layer.check()
    ok, msg = oracle.check_moe_output(y, oracle.moe_expected_output(cfg, data, 1))
    assert ok, msg
    d, c = layer.trace[0].tolist(), layer.trace[1].tolist()
    assert all(v > 0 for v in d) and d[:7] == sorted(d[:7]) and d[7] >= d[6]  # dispatch phases in order
    assert c[0] > 0 and c[7] >= c[2] >= c[1] >= c[0] and c[0] >= d[0]
    layer.close()


@pytest.mark.parametrize("mode", ["dedup", "direct"])
def test_moe_combine_accepts_foreign_expert_y(mode):
    from amd_distributed_2025_b200.models import moe_all2all

    cfg, data, _, _ = contract.make_moe_inputs(32, 4, 512, 64, 3, 0, 1, device="cuda", fixed_num_tokens=64)
    layer = moe_all2all.get_layer(cfg, 0, 1, mode=mode)
    n_tok, ex, em = layer.dispatch(data.x, data.indices)
    ey = ex.clone() * 3  # an ordinary tensor, not the symmetric buffer
    y = torch.zeros(cfg.max_num_tokens, cfg.hidden_dim, dtype=cfg.out_dtype, device="cuda")
    layer.combine(y, data.weights, em, ey, n_tok, data.num_tokens)
    torch.cuda.synchronize()
    want = (data.x.float() * 3 * data.weights.sum(1, keepdim=True)).to(cfg.out_dtype)
    assert torch.allclose(y[: data.num_tokens].float(), want.float(), rtol=1e-2, atol=5e-3)


@pytest.mark.parametrize("mode", ["dedup", "direct"])
def test_moe_bad_expert_id_is_reported_not_faulted(mode):
    from amd_distributed_2025_b200.models import moe_all2all
    from amd_distributed_2025_b200.utils.status import StatusError

    cfg, data, _, _ = contract.make_moe_inputs(16, 2, 128, 8, 3, 0, 1, device="cuda", fixed_num_tokens=8)
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode=mode)
    bad = data.indices.clone()
    bad[2, 1] = 99
    y = layer.forward(data.x, bad, data.weights, 2.0)
    torch.cuda.synchronize()
    with pytest.raises(StatusError) as err:
        layer.check()
    assert err.value.code == "bad_index"
    # the other entries were served: every token but the one with the bad id has its full result
    want = (data.x.float() * 2 * data.weights.sum(1, keepdim=True)).to(cfg.out_dtype)
    keep = [t for t in range(8) if t != 2]
    assert torch.allclose(y[keep].float(), want[keep].float(), rtol=1e-2, atol=5e-3)
    layer.ws.reset_status()
    layer.close()


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("H", [64, 65])  # rows of whole vectors, and not
def test_moe_one_rank_entries_that_do_not_fit_their_expert(fused, H):
    """A token that names an expert twice can send it more rows than the layer has room for: the others are delivered,
    and the record says which entry had which slot."""
    from amd_distributed_2025_b200.models import moe_all2all
    from amd_distributed_2025_b200.utils.status import StatusError

    T, k = 4, 8  # room for four rows an expert
    cfg = contract.MoEConfig(2, k, H, T, torch.float32, torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(T, H, device="cuda", generator=gen)
    w = torch.rand(T, k, device="cuda", generator=gen)
    ids = torch.zeros(T, k, dtype=torch.int32, device="cuda")  # expert 0: entry i is its row i ...
    ids[1, 6] = ids[3, 7] = 1  # ... but for two that go to expert 1, after which it is row i - 1
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
    assert layer.max_recv == T
    if fused:
        y = layer.forward(x, ids, w, 2.0)
        served = torch.zeros(T, k, dtype=torch.float64, device="cuda")
        served[0, :4] = served[1, 6] = served[3, 7] = 1.0
        want = 2.0 * x.double() * (w.double() * served).sum(1, keepdim=True)
        assert oracle.relative_error(y, want) < 1e-6
        counts, ex, meta = layer.expert_num_tokens, layer.expert_x, layer.expert_meta
    else:
        counts, ex, meta = layer.dispatch(x, ids)
    with pytest.raises(StatusError) as err:
        layer.check()
    entry, slot = err.value.status["detail"], err.value.status["seen"]
    assert err.value.code == "bad_index" and 4 <= entry < 31 and entry != 14 and slot == entry - (entry > 14)
    assert counts.tolist() == [4, 2]
    assert torch.equal(ex[0], x[[0, 0, 0, 0]]) and torch.equal(ex[1, :2], x[[1, 3]])
    assert meta[0].tolist() == [[0, 0, 0, j, 0] for j in range(4)] and meta[1, :2].tolist() == [[1, 0, 1, 6, 0], [1, 0, 3, 7, 0]]
    layer.ws.reset_status()
    layer.close()


@pytest.mark.parametrize(
    "m,n,k,has_bias",
    [
        (128, 256, 64, False),      # one tile, one k-block
        (128, 256, 512, True),
        (256, 512, 1024, True),
        (64, 2880, 360, True),      # ragged M, N and K (K/8 of the smallest task shape)
        (2048, 5120, 1600, True),
        (512, 4608, 4608, False),
        (1024, 8192, 3584, True),
    ],
)
def test_gemm_world1_matches_fp32_reference(m, n, k, has_bias):
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, has_bias, 5, device="cuda")
    out = gemm_rs.custom_kernel((a, w, bias))
    torch.cuda.synchronize()
    gemm_rs.get_op(m, n, k).check()
    truth = a.float() @ w.float().T
    if has_bias:
        truth = truth + bias.float()
    want = oracle.gemm_rs_fused_rounding([a], [w], bias, 0)
    assert oracle.outlier_fraction(out, want, oracle.GEMM_RS_RTOL, oracle.GEMM_RS_ATOL) < 1e-4
    assert oracle.relative_error(out, truth) < 5e-3


@pytest.mark.parametrize(
    "m,n,k",
    [
        (1, 512, 64),  # one token, one k-block
        (33, 520, 1032),  # ragged in all three: rows of W start between cache lines
        (30, 512, 29568),  # a few tiles, K shared by a large cluster
        (90, 2048, 2752),  # ... by a small one
        (256, 5120, 6400),  # CTA pairs, two of them to a tile
        (700, 2208, 1112),  # CTA pairs, one tile each; several along M, short last ones
        (129, 8192, 264),  # one row more than a tile: swapped, on pairs
        (2048, 2880, 2880),  # persistent pairs, whole tiles
        (2560, 4096, 1032),  # ... ragged along K
        (4162, 1248, 4280),  # ... and tiles cut along K, ragged
        (3000, 3000, 512),
        (7990, 7688, 12296),  # tiles of two accumulators, the last ones ragged
    ],
)
def test_gemm_one_rank_schedules(m, n, k):
    """Every schedule of the one-rank kernels against fp32, with both orders of the bias, call after call."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 17, device="cuda")
    op = gemm_rs.get_op(m, n, k)
    truth = a.float() @ w.float().T
    cases = [(None, "per_rank", truth), (bias, "per_rank", truth.bfloat16().float() + bias.float()),
             (bias, "once", truth + bias.float())]
    for b, mode, want in cases:
        first = op(a, w, b, mode)
        for _ in range(3):
            again = op(a, w, b, mode)
        torch.cuda.synchronize()
        op.check()
        assert torch.equal(first, again)
        assert oracle.relative_error(first, want) < 5e-3
        assert float((first.float() - want).abs().max()) < 1e-2 * float(want.abs().max())


@pytest.mark.parametrize(
    "kind,m,n,k",
    [  # kernel, which operand has the 128 rows, CTAs, where the parts of a shared tile meet / accumulators / cut tiles
        ("tile normal single", 202, 656, 256),
        ("tile normal single shared own", 4, 512, 1152),
        ("tile normal single shared pipeline", 1058, 624, 3104),
        ("tile normal pair", 386, 688, 328),
        ("tile normal pair shared own", 388, 736, 912),
        ("tile normal pair shared pipeline", 1528, 528, 5152),
        ("tile swapped single", 1, 512, 256),
        ("tile swapped single shared own", 1, 512, 904),
        ("tile swapped single shared pipeline", 67, 1856, 3880),
        ("tile swapped pair", 206, 1168, 344),
        ("tile swapped pair shared own", 1, 4416, 5792),
        ("tile swapped pair shared pipeline", 632, 512, 5384),
        ("pair normal", 1822, 3352, 104),
        ("pair normal cut", 1180, 4088, 2584),
        ("pair normal two accumulators", 4759, 5240, 4424),  # three waves
        ("pair normal two accumulators", 3441, 1944, 3344),
        ("pair swapped", 411, 7280, 256),
        ("pair swapped cut", 522, 7568, 1936),
        ("pair swapped two accumulators", 2551, 6744, 3984),  # two waves
        ("pair swapped two accumulators", 1465, 4688, 3816),
    ],
)
def test_gemm_one_rank_reaches_every_path(kind, m, n, k):
    """One size for every path that the one-rank planner takes, ragged against its tiles.  Bounds as derived for
    one rounding of an fp32 sum to bf16 (2^-9 relative), twice where a bias is added to the rounded product."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 23, device="cuda")
    op = gemm_rs.get_op(m, n, k)
    truth = a.double() @ w.double().T
    for b, mode, want in ((None, "per_rank", truth), (bias, "per_rank", truth.bfloat16().double() + bias.double()),
                          (bias, "once", truth + bias.double())):
        first = op(a, w, b, mode)
        assert torch.equal(first, op(a, w, b, mode))
        op.check()
        assert oracle.relative_error(first, want) < 5e-3
        assert float((first.double() - want).abs().max()) < 1e-2 * float(want.abs().max())
    p = _ext().gemm_local_plan(m, n, k, torch.cuda.get_device_properties(0).multi_processor_count)
    got = [p["kernel"], "swapped" if p["swap"] else "normal"]
    if p["kernel"] == "tile":
        got.append("pair" if p["cta_pair"] else "single")
        if p["splits"] > 1:
            got += ["shared", "own" if p["own_parts"] else "pipeline"]
    else:
        got += ["cut"] * (p["cut_tiles"] > 0) + ["two accumulators"] * (p["halves"] == 2)
    _check_plan(" ".join(got), kind)


@pytest.mark.parametrize(
    "kind,m,n,k",
    [
        ("tile normal single", 206, 4792, 64),  # one k-block; the last column tile holds 88 of 96 columns
        ("tile normal single shared own", 384, 1040, 1736),
        ("tile normal single shared pipeline", 362, 744, 3472),
        ("tile normal pair", 242, 4760, 264),
        ("tile normal pair shared own", 396, 1040, 2088),
        ("tile normal pair shared pipeline", 646, 1104, 2952),  # three parts of 160 columns: 56, 56 and 48 to finish
        ("pair normal", 7639, 520, 72),
        ("pair normal", 2048, 2880, 2880),  # 160 columns: five chunks, three for one half of the warps
        ("pair normal cut", 6345, 656, 1888),  # 224 columns, left in the workspace chunk by chunk
    ],
)
def test_gemm_one_rank_widths_of_an_odd_number_of_chunks(kind, m, n, k):
    """Tiles of 96, 160 and 224 columns, whose groups leave chunk by chunk."""
    test_gemm_one_rank_reaches_every_path(kind, m, n, k)
    assert _ext().gemm_local_plan(m, n, k, _PART[0])["bn"] % 64 == 32


@pytest.mark.parametrize(
    "kind,m,n,k",
    [
        ("tile normal single", 134, 1040, 256),
        ("tile normal single shared pipeline", 1088, 608, 2600),
        ("tile normal pair shared own", 389, 768, 848),
        ("pair normal", 5477, 712, 256),
    ],
)
def test_gemm_one_rank_reaches_the_widths_of_whole_groups(kind, m, n, k):
    """The same paths at multiples of 64 columns."""
    test_gemm_one_rank_reaches_every_path(kind, m, n, k)
    assert _ext().gemm_local_plan(m, n, k, _PART[0])["bn"] % 64 == 0


@pytest.mark.parametrize("m,n,k", [
    (2048, 2880, 2880), (6345, 656, 1888), (4759, 5240, 4424), (242, 4760, 264), (134, 1040, 256), (646, 1104, 2952),  # normal
    (411, 7280, 256), (206, 1168, 344),  # swapped
])
def test_gemm_one_rank_bias_is_added_to_the_rounded_product(m, n, k):
    """Bit for bit what the library's bf16 addition makes of the product without a bias."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 29, device="cuda")
    bias = (bias.float() * 2.0 ** torch.randint(-30, 8, bias.shape, device="cuda").float()).bfloat16()
    op = gemm_rs.get_op(m, n, k)
    plain = op(a, w, None)
    assert torch.equal(op(a, w, bias, "per_rank"), plain + bias)
    op.check()


def test_gemm_one_rank_bias_of_every_kind_of_number():
    """Products and bias values of every bit pattern, infinities, NaNs, signed zeros and subnormal numbers among them."""
    from amd_distributed_2025_b200.models import gemm_rs

    m, n, k = 256, 8192, 64
    gen = torch.Generator(device="cuda").manual_seed(3)
    a = torch.zeros(m, k, dtype=torch.bfloat16, device="cuda")
    a[:, 0] = 1.0
    for _ in range(4):
        w = torch.zeros(n, k, dtype=torch.bfloat16, device="cuda")
        w[:, 0] = torch.randint(-32768, 32768, (n,), device="cuda", generator=gen).short().view(torch.bfloat16)
        bias = torch.randint(-32768, 32768, (n,), device="cuda", generator=gen).short().view(torch.bfloat16)
        near = torch.rand(n, device="cuda", generator=gen) < 0.5  # exponents that are close, or the sum is one of the two
        bias = torch.where(near, (w[:, 0].float() * -1.007).bfloat16(), bias)
        op = gemm_rs.get_op(m, n, k)
        want = op(a, w, None) + bias
        got = op(a, w, bias, "per_rank")
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.equal(got[~want.isnan()].view(torch.int16), want[~want.isnan()].view(torch.int16))


@pytest.mark.parametrize("m,n,k,has_bias", [(64, 2880, 360, True), (512, 4096, 1536, True), (2048, 2880, 360, True)])
def test_gemm_world1_reference_inputs_pass_reference_checker(m, n, k, has_bias):
    """Operands from the reference generator (uniform +-0.01) against the library path."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.generate_gemm_rs_input(0, 1, m, n, k, has_bias, 2035, device="cuda")
    out = gemm_rs.custom_kernel((a, w, bias))
    ref = torch.matmul(a, w.T) + bias
    ok, msg = oracle.check_gemm_rs_output(out, ref)
    assert ok, msg
    truth = a.double() @ w.double().T + bias.double()
    assert oracle.relative_error(out, truth) < 5e-3


@pytest.mark.parametrize(
    "m,n,k,block_n,cta_pair,splits",
    [(*size, *tile) for size in ((384, 1024, 832), (128, 256, 64), (1000, 2880, 360), (2048, 2048, 2048))
     for tile in ((64, 0, 1), (128, 0, 1), (256, 0, 1), (128, 1, 1), (192, 1, 1), (256, 1, 1), (256, 1, 3), (192, 1, 2), (128, 0, 4))
     if tile[2] <= (size[2] + 63) // 64])  # (no more K slices than k-blocks)
def test_gemm_tile_shapes_single_cta_and_cta_pair(m, n, k, block_n, cta_pair, splits):
    """Every tile width, as single CTAs and as CTA pairs (256-row tiles, odd block counts
    and ragged edges included), gives the same GEMM."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 9, device="cuda")
    op = gemm_rs.get_op(m, n, k)
    op.block_n, op.cta_pair, op.splits = block_n, cta_pair, splits
    try:
        for _ in range(3):  # staged paths alternate parities and reset their counters
            out = op(a, w, bias)
        torch.cuda.synchronize()
        op.check()
    finally:
        op.block_n, op.cta_pair, op.splits = 0, -1, 0
    truth = a.float() @ w.float().T + bias.float()
    assert oracle.relative_error(out, truth) < 5e-3
    want = oracle.gemm_rs_fused_rounding([a], [w], bias, 0)
    assert oracle.outlier_fraction(out, want, oracle.GEMM_RS_RTOL, oracle.GEMM_RS_ATOL) < 1e-4


@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (256, 384, 512), (1000, 2944, 1024), (4096, 4096, 2048)])
def test_fp8_block_scaled_gemm_matches_fp32_reference(m, n, k):
    from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm, fp8_gemm_reference

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    b = torch.randn(n, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    kb, nb = (k + 127) // 128, (n + 127) // 128
    # scales stored the way the stand-alone template indexes them: [kb][m] and [kb][nb], viewed transposed
    a_scale = (torch.rand(kb, m, device="cuda", generator=g) + 0.5).t()
    b_scale = (torch.rand(kb, nb, device="cuda", generator=g) + 0.5).t()
    c = fp8_gemm(a, b, a_scale, b_scale)
    torch.cuda.synchronize()
    want = fp8_gemm_reference(a, b, a_scale, b_scale)
    assert oracle.relative_error(c, want) < 5e-3
    assert torch.allclose(c.float(), want, rtol=2e-2, atol=2e-2 * float(want.abs().max()))


@pytest.mark.parametrize("m,n,k", [(1, 8, 16), (257, 200, 1040), (64, 1024, 4096), (200, 264, 1280), (300, 619, 400), (129, 136, 1408), (4100, 3000, 640)])
def test_fp8_gemm_schedules(m, n, k):
    """Shared and whole tiles, ragged rows, columns and K, scales by rows (four at a time where aligned), with and without ``c``."""
    from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm, fp8_gemm_reference

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    b = torch.randn(n, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    a_scale = torch.rand(m, (k + 127) // 128, device="cuda", generator=g) + 0.5
    b_scale = torch.rand((n + 127) // 128, (k + 127) // 128, device="cuda", generator=g) + 0.5
    out = fp8_gemm(a, b, a_scale, b_scale)
    again = fp8_gemm(a, b, a_scale, b_scale, c=torch.empty_like(out))
    want = fp8_gemm_reference(a, b, a_scale, b_scale)
    assert torch.equal(out, again)
    assert oracle.relative_error(out, want) < 5e-3
    assert float((out.float() - want).abs().max()) < 1e-2 * float(want.abs().max())


@pytest.mark.parametrize(
    "bn,splits,m,n,k",
    [
        (64, 1, 2638, 784, 144),  # several waves; two K blocks, the second one ragged
        (64, 2, 788, 326, 3408),
        (64, 4, 518, 179, 2032),
        (64, 5, 154, 120, 1840),  # 16 columns for each of the five, but none for the last
        (64, 7, 129, 112, 2384),  # one row in the second CTA of the pair
        (64, 8, 176, 110, 2944),
        (128, 1, 361, 2824, 176),
        (128, 1, 3687, 1096, 144),  # several waves
        (128, 1, 2803, 1556, 16),  # part of a K block
        (128, 2, 270, 1896, 5824),
        (128, 3, 139, 2335, 5088),  # 48, 48 and 32 columns to finish; rows of C are no whole 16-byte pieces
        (128, 4, 338, 750, 5440),
    ],
)
def test_fp8_gemm_narrow_tiles(bn, splits, m, n, k):
    """Tiles of 64 and 128 columns, whole and shared."""
    _fp8_gemm_against_fp64(m, n, k)
    _check_plan(_ext().fp8_gemm_plan(m, n, k, _PART[0]), (bn, splits))


@pytest.mark.parametrize(
    "bn,m,n,k",
    [
        (192, 1000, 3003, 656),  # one wave: rows and columns end inside a tile, rows of C are no whole 16-byte pieces
        (192, 2100, 4104, 1040),  # several waves, the last column tile an eighth full; nine K blocks
        (256, 640, 5003, 656),
        (256, 257, 9000, 400),  # one row in the second row of tiles; four K blocks: one set of scales
        (256, 3000, 5904, 528),  # several waves, five K blocks: one of them in a set of its own
        (256, 1118, 6664, 128),  # one K block, several waves
    ],
)
def test_fp8_gemm_wide_tiles(bn, m, n, k):
    """Tiles of 192 and 256 columns."""
    _fp8_gemm_against_fp64(m, n, k)
    _check_plan(_ext().fp8_gemm_plan(m, n, k, _PART[0]), (bn, 1))


def _fp8_gemm_against_fp64(m, n, k):
    """A sum rounds once to bf16 (2^-9 of it at most); partial sums are fp32."""
    from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    b = torch.randn(n, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    kb = (k + 127) // 128
    a_scale = torch.rand(m, kb, device="cuda", generator=g) + 0.5
    b_scale = torch.rand((n + 127) // 128, kb, device="cuda", generator=g) + 0.5
    out = fp8_gemm(a, b, a_scale, b_scale)
    spread = torch.arange(k, device="cuda") // 128
    want = (a.double() * a_scale.double()[:, spread]) @ (b.double() * b_scale.double().repeat_interleave(128, 0)[:n, spread]).T
    assert torch.equal(out, fp8_gemm(a, b, a_scale, b_scale))
    assert oracle.relative_error(out, want) < 2.0**-9
    assert float(((out.double() - want).abs() - want.abs() * 2.0**-8).max()) < 1e-4 * float(want.abs().max())


@pytest.mark.parametrize("tma_store", [True, False])
@pytest.mark.parametrize("fuse_own", [True, False])
@pytest.mark.parametrize("m,n,k,block_n,cta_pair", [(2048, 2048, 1024, 256, 1), (1024, 2880, 512, 192, 1), (512, 1024, 256, 128, 0),
                                                   (1056, 1000, 320, 256, 1)])
def test_gemm_staged_path_on_one_gpu(tma_store, fuse_own, m, n, k, block_n, cta_pair):
    """The multi-rank machinery (staging buffer, TMA stores, signaller, arrival counters,
    reduction) run on a single rank, where its result must equal the plain GEMM."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 13, device="cuda")
    op = gemm_rs.get_op(m, n, k)
    op.block_n, op.cta_pair, op.splits = block_n, cta_pair, 1
    op.force_staged, op.tma_store, op.fuse_own = True, tma_store, fuse_own
    try:
        for _ in range(3):
            out = op(a, w, bias)
        torch.cuda.synchronize()
        op.check()
    finally:
        op.block_n, op.cta_pair, op.splits = 0, -1, 0
        op.force_staged, op.tma_store, op.fuse_own = False, True, None
    want = oracle.gemm_rs_fused_rounding([a], [w], bias, 0)
    assert oracle.outlier_fraction(out, want, oracle.GEMM_RS_RTOL, oracle.GEMM_RS_ATOL) < 1e-4
    assert oracle.relative_error(out, a.float() @ w.float().T + bias.float()) < 5e-3


def test_closed_operators_launch_nothing():
    """After close() there is no slab and no status record: native entry points refuse by themselves, whoever holds them."""
    from amd_distributed_2025_b200.models import gemm_rs, moe_all2all

    cfg, data, _, _ = contract.make_moe_inputs(16, 2, 256, 8, 3, 0, 1, device="cuda", fixed_num_tokens=8)
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
    engine, heap, y = layer.engine, layer.ws.heap, torch.zeros(8, 256, dtype=cfg.out_dtype, device="cuda")
    ey = torch.zeros(layer.expert_y.shape, dtype=cfg.out_dtype, device="cuda")
    layer.forward(data.x, data.indices, data.weights, 1.0)
    layer.close()
    assert engine.try_forward(data.x, data.indices, data.weights, 1.0) is None
    assert not engine.try_dispatch(data.x, data.indices) and not engine.try_combine(y, data.weights, ey, 8)
    for call in (lambda: engine.forward(data.x, data.indices, data.weights, y, 1.0), lambda: engine.dispatch(data.x, data.indices),
                 lambda: engine.combine(y, data.weights, ey), lambda: heap.view(4096, [16], torch.uint8),
                 lambda: heap.barrier(1, 1000), lambda: heap.wait_selftest(0, 1, 1000),
                 lambda: layer.forward(data.x, data.indices, data.weights, 1.0)):
        with pytest.raises(RuntimeError):
            call()
    a, w, bias = contract.make_gemm_rs_inputs(0, 1, 64, 512, 256, True, 5, device="cuda")
    op = gemm_rs.GemmRS(1 << 20, 1 << 12, rank=0, world_size=1)
    op(a, w, bias)
    op.close()
    assert op.engine.try_run(a, w, bias, True) is None
    with pytest.raises(RuntimeError):
        op(a, w, bias)
    torch.cuda.synchronize()
    assert float(torch.ones(4, device="cuda").sum()) == 4.0


@pytest.mark.parametrize("m,n,k", [(32, 136, 1000), (8, 64, 1024), (17, 128, 904)])
def test_gemm_small_clusters_of_two_streams_share_sms(m, n, k):
    """Tiles so small that CTAs of two launches meet on an SM: both find their tensor memory there."""
    from amd_distributed_2025_b200.models import gemm_rs

    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 3, device="cuda")
    op = gemm_rs.get_op(m, n, k)
    want = op(a, w, bias)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for _ in range(50):
        for s in streams:
            with torch.cuda.stream(s):
                outs.append(op(a, w, bias))
    torch.cuda.synchronize()
    op.check()
    assert all(torch.equal(o, want) for o in outs)
    assert oracle.relative_error(want, (a.float() @ w.float().T).bfloat16().float() + bias.float()) < 5e-3


@pytest.mark.parametrize("clear", ["reset_status", "recover"])
def test_workspace_of_cut_tiles_does_not_outlive_a_failure(clear):
    """A kernel that gave up may leave a tile's counter behind; the next call must not take it for its other half."""
    from amd_distributed_2025_b200.models import gemm_rs

    m, n, k = 4162, 1248, 4280  # tiles cut along K
    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 17, device="cuda")
    op = gemm_rs.GemmRS(1 << 20, 1 << 12, rank=0, world_size=1)
    want = op(a, w, bias)
    (old,) = op.engine.local_workspaces()
    assert torch.equal(op(a, w, bias), want) and op.engine.local_workspaces()[0].data_ptr() == old.data_ptr()
    op.ws.reset_status() if clear == "reset_status" else op.recover()
    assert torch.equal(op(a, w, bias), want)
    (new,) = op.engine.local_workspaces()
    assert new.data_ptr() != old.data_ptr()
    op.check()
    op.close()


def test_fp8_gemm_expired_wait_leaves_a_record():
    from amd_distributed_2025_b200.ops import fp8_gemm as f
    from amd_distributed_2025_b200.utils.status import StatusError

    ext = _ext()
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(128, 256, device="cuda", generator=g).to(torch.float8_e4m3fn)
    s = torch.ones(128, 2, device="cuda")
    want = f.fp8_gemm(a, a, s, s[:1])
    f.check()
    for ask in (f.check, lambda: f.fp8_gemm(a, a, s, s[:1]), lambda: f.fp8_gemm(a, a, s, s[:1], c=torch.empty_like(want))):
        ext.fp8_wait_selftest(0, 1_000_000)  # a barrier nobody arrives on, 1 ms
        torch.cuda.synchronize()
        with pytest.raises(StatusError) as err:
            ask()
        assert err.value.code == "timeout" and err.value.phase == "gemm_pipeline" and err.value.status["detail"] == 900
        assert torch.equal(f.fp8_gemm(a, a, s, s[:1]), want)
        f.check()


def test_fp8_gemm_first_call_of_a_process_may_be_captured():
    """Nothing that the first call sets up (opt-ins, plan, the record's memory) breaks a capture off."""
    import os
    import subprocess
    import sys

    code = """
import torch
from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm, fp8_gemm_reference
a = torch.randn(256, 512, device="cuda").to(torch.float8_e4m3fn)
s, t = torch.rand(256, 4, device="cuda"), torch.rand(2, 4, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    c = fp8_gemm(a, a, s, t)
graph.replay()
torch.cuda.synchronize()
want = fp8_gemm_reference(a, a, s, t)
assert float((c.float() - want).abs().max()) < 1e-2 * float(want.abs().max())
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def _captured_case(op, size):
    """(buffers to refill, how to fill them, the call) of a one-rank operator."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    normal = lambda *shape, dtype=torch.float32: torch.randn(*shape, device="cuda", generator=gen).to(dtype)  # noqa: E731
    if op.startswith("moe"):
        from amd_distributed_2025_b200.models import moe_all2all

        E, k, H, T = size
        cfg, data, _, _ = contract.make_moe_inputs(E, k, H, T, 5, 0, 1, device="cuda", dtype=torch.bfloat16, fixed_num_tokens=T)
        layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="dedup")
        bufs = [data.x, data.indices, data.weights]
        fill = lambda: [normal(T, H, dtype=torch.bfloat16), torch.argsort(normal(T, E), 1)[:, :k].int(), normal(T, k)]  # noqa: E731
        if op == "moe_forward":
            return bufs, fill, lambda: [layer.forward(*bufs, 3.0)], layer
        out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")

        def layered():
            counts, ex, meta = layer.dispatch(bufs[0], bufs[1])
            layer.combine(out, bufs[2], meta, ex, counts, T)
            return [out, counts]

        return bufs, fill, layered, layer
    m, n, k = size
    if op == "fp8":
        from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm

        fill = lambda: [normal(m, k).to(torch.float8_e4m3fn), normal(n, k).to(torch.float8_e4m3fn),  # noqa: E731
                        normal(m, (k + 127) // 128), normal((n + 127) // 128, (k + 127) // 128)]
        bufs = fill()
        return bufs, fill, lambda: [fp8_gemm(*bufs)], None
    from amd_distributed_2025_b200.models import gemm_rs

    gemm = gemm_rs.GemmRS(1 << 20, 1 << 12, rank=0, world_size=1)
    fill = lambda: [normal(m, k, dtype=torch.bfloat16), normal(n, k, dtype=torch.bfloat16), normal(n, dtype=torch.bfloat16)]  # noqa: E731
    bufs = fill()
    return bufs, fill, lambda: [gemm(*bufs), gemm(*bufs, bias_mode="once")], gemm


@pytest.mark.parametrize(
    "op,size",
    [
        ("moe_forward", (64, 4, 512, 96)),
        ("moe_layer", (64, 4, 512, 96)),
        ("gemm", (64, 2880, 360)),  # clusters that share a tile
        ("gemm", (4162, 1248, 4280)),  # tiles cut along K, which meet in a workspace of the graph's own
        ("fp8", (300, 619, 400)),
    ],
)
def test_one_rank_operators_replayed_from_graphs(op, size):
    """Captured once, replayed with other inputs, on another stream, and with calls outside the graph in between."""
    bufs, fill, call, owner = _captured_case(op, size)
    call()
    graphs = []
    for _ in range(6):  # more graphs than the GEMM keeps workspaces for
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs = call()
        graphs.append((g, outs))
    side = torch.cuda.Stream()
    for turn, (g, outs) in enumerate(graphs + graphs[:2]):
        for b, v in zip(bufs, fill()):
            b.copy_(v)
        if turn % 2:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                g.replay()
                g.replay()
            torch.cuda.current_stream().wait_stream(side)
        else:
            g.replay()
        got = [o.clone() for o in outs]
        want = call()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), turn
    if owner is not None:
        owner.check()
        owner.close()


def test_gemm_cut_tiles_on_more_streams_than_workspaces():
    """Calls on several streams at once: the first four streams get a workspace each, the others run whole tiles."""
    from amd_distributed_2025_b200.models import gemm_rs

    m, n, k = 4162, 1248, 4280
    a, w, bias = contract.make_gemm_rs_inputs(0, 1, m, n, k, True, 17, device="cuda")
    op = gemm_rs.GemmRS(1 << 20, 1 << 12, rank=0, world_size=1)
    cut = op(a, w, bias, "once")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(6)]
    outs = [[] for _ in streams]
    for _ in range(4):
        for s, got in zip(streams, outs):
            with torch.cuda.stream(s):
                got.append(op(a, w, bias, "once"))
    torch.cuda.synchronize()
    op.check()
    assert len(op.engine.local_workspaces()) == 4
    truth = a.float() @ w.float().T + bias.float()
    for i, got in enumerate(outs):
        assert all(torch.equal(o, got[0]) for o in got)
        assert i >= 3 or torch.equal(got[0], cut)
        assert oracle.relative_error(got[0], truth) < 5e-3
    op.close()


def test_host_tensors_are_refused_before_a_launch():
    """A kernel that is given the address of an ordinary host tensor faults: scales, bias, results, weights, expert rows."""
    from amd_distributed_2025_b200.models import gemm_rs, moe_all2all
    from amd_distributed_2025_b200.ops.fp8_gemm import fp8_gemm

    a = torch.ones(128, 256, device="cuda").to(torch.float8_e4m3fn)
    s, t = torch.ones(128, 2, device="cuda"), torch.ones(1, 2, device="cuda")
    x, w, bias = contract.make_gemm_rs_inputs(0, 1, 64, 512, 256, True, 5, device="cuda")
    op = gemm_rs.get_op(64, 512, 256)
    cfg, data, _, _ = contract.make_moe_inputs(16, 2, 256, 8, 3, 0, 1, device="cuda", fixed_num_tokens=8)
    layer = moe_all2all.MoEAllToAll(cfg, 0, 1, mode="direct")
    counts, ex, meta = layer.dispatch(data.x, data.indices)
    y = torch.empty(8, 256, dtype=cfg.out_dtype, device="cuda")
    for call in (lambda: fp8_gemm(a, a, s.cpu(), t), lambda: fp8_gemm(a, a, s, t.cpu()),
                 lambda: fp8_gemm(a, a, s, t, c=torch.empty(128, 128, dtype=torch.bfloat16)),
                 lambda: op(x, w, bias.cpu()), lambda: op(x, w, bias, out=torch.empty(64, 512, dtype=torch.bfloat16)),
                 lambda: layer.combine(y, data.weights.cpu(), meta, ex, counts), lambda: layer.combine(y, data.weights, meta, ex.cpu(), counts)):
        with pytest.raises(RuntimeError):
            call()
    want = op(x, w, bias)
    assert torch.equal(op(x, w, bias.cpu().pin_memory()), want)  # memory that the GPU can read stays accepted
    torch.cuda.synchronize()
    layer.check()
    layer.close()


def test_gemm_stamps_stay_inside_the_trace_tensor():
    """A grid of several waves has more CTAs than the trace has rows: it leaves no stamps then."""
    from amd_distributed_2025_b200.models import gemm_rs

    op = gemm_rs.GemmRS(1 << 20, 1 << 12, rank=0, world_size=1)
    buf = torch.zeros(2048, 8, dtype=torch.int64, device="cuda")
    op.engine.set_trace(buf[:160])  # (any CTA's row would lie in `buf`)
    m, n, k = 16, 32000, 4096
    plan = _ext().gemm_local_plan(m, n, k, torch.cuda.get_device_properties(0).multi_processor_count)
    assert 160 < plan["ctas"] <= 2048
    a, w, _ = contract.make_gemm_rs_inputs(0, 1, m, n, k, False, 1, device="cuda")
    op(a, w)
    torch.cuda.synchronize()
    assert int(buf.abs().sum()) == 0
    op.engine.set_trace(buf)
    op(a, w)
    torch.cuda.synchronize()
    assert bool((buf[: plan["ctas"], :4] > 0).all()) and int(buf[plan["ctas"]:].abs().sum()) == 0
    op.close()

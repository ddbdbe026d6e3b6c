"""Routes that a rule on sizes picks, against the general route of the same call: the same bits."""
import re

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from owoinfer_b200 import ops as o
    return o


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _kernels(call):
    """The (mangled) names of the kernels that a call launches, in order of capture."""
    from cuda.bindings import driver as cu
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1:]
    handle = cu.CUgraph(graph.raw_cuda_graph())
    names = []
    for node in ok(cu.cuGraphGetNodes(handle, ok(cu.cuGraphGetNodes(handle, 0))[1]))[0]:
        if ok(cu.cuGraphNodeGetType(node))[0] == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(cu.cuGraphKernelNodeGetParams(node))[0]
            name = cu.cuFuncGetName(params.func) if int(params.func) else cu.cuKernelGetName(params.kern)
            names.append(ok(name)[0].decode())
    return names


@pytest.mark.parametrize("m", [1, 127, 256, 257, 297, 384, 512])
@pytest.mark.parametrize("n,k", [(64, 512), (1000, 528), (3072, 3072), (3064, 8192)])
def test_gemm_tiles_that_share_k_give_the_bits_of_whole_tiles(ops, m, n, k):
    """Few rows: AUTO takes tiles whose K range a cluster shares where whole ones would leave SMs idle. Edges: one row, the
    edges of 128- and 256-row tiles, columns that end inside a 64-column unit, K blocks that do not divide evenly."""
    g = _gen(m * 7 + n + k)
    x = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    xs, ws = torch.rand(m, device="cuda", generator=g) * 1e-3, torch.rand(n, device="cuda", generator=g) * 1e-3
    bias, gate = (torch.randn(n, device="cuda", generator=g).bfloat16() for _ in range(2))
    res = torch.randn((m, n), device="cuda", generator=g).bfloat16()
    want, want_res = ops.int8_gemm(x, xs, w, ws, bias, tile=ops.TILE_128x128), res.clone()
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, want_res, tile=ops.TILE_128x128)
    got = ops.int8_gemm(x, xs, w, ws, bias)
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, res)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(res.view(torch.int16), want_res.view(torch.int16))
    assert ops.kernel_status() == (0, 0)


def _gemm_route(call):
    """(tile columns, CTAs of a tile, CTAs or pairs that share its K range) of the one INT8 GEMM kernel that a call launches."""
    name, = _kernels(call)
    return tuple(int(v) for v in re.search(r"int8_gemm_kernelILi(\d+)E.*?ELi(\d)ELb0ELi(\d)E", name).groups())


# Both ends of a tile's rows, columns that end inside a 64-column unit, K blocks that the CTAs of a cluster cannot share evenly (65,
# 97, 17 of them), and a last K block that is not full.
SHARED_K = [(1, 3064, 8208, (128, 1, 2)), (257, 3072, 3088, (128, 1, 2)), (384, 3064, 8208, (128, 1, 2)), (100, 1000, 2064, (128, 1, 2)),
            (128, 9216, 3072, (128, 1, 2)), (385, 3064, 8208, (256, 2, 2)), (400, 3064, 12304, (256, 2, 2)), (512, 3072, 8208, (256, 2, 2)),
            (1, 3064, 12288, (256, 2, 4)), (129, 2056, 16400, (256, 2, 4)), (256, 3072, 12304, (256, 2, 4))]


@pytest.mark.parametrize("m,n,k,route", SHARED_K)
def test_each_way_of_sharing_k_gives_the_bits_of_whole_tiles(ops, m, n, k, route):
    """The three cluster shapes that AUTO takes for few rows, by the kernel that is launched: plain, column-chunked and
    gated-residual outputs against whole 128 x 128 tiles."""
    g = _gen(m * 7 + n + k)
    x = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    xs, ws = torch.rand(m, device="cuda", generator=g) * 1e-3, torch.rand(n, device="cuda", generator=g) * 1e-3
    bias, gate = (torch.randn(n, device="cuda", generator=g).bfloat16() for _ in range(2))
    res = torch.randn((m, n), device="cuda", generator=g).bfloat16()
    want, want_res = ops.int8_gemm(x, xs, w, ws, bias, tile=ops.TILE_128x128), res.clone()
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, want_res, tile=ops.TILE_128x128)
    chunk = n // 8 if n % 64 == 0 else n
    got, chunks, out_res = ops.int8_gemm(x, xs, w, ws, bias), ops.int8_gemm_chunked(x, xs, w, ws, chunk, bias=bias), res.clone()
    ops.int8_gemm_gated_residual(x, xs, w, ws, gate, out_res)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(chunks.permute(1, 0, 2).reshape(m, n).view(torch.int16), want.view(torch.int16))
    assert torch.equal(out_res.view(torch.int16), want_res.view(torch.int16))
    assert ops.kernel_status() == (0, 0)
    scratch = res.clone()
    assert _gemm_route(lambda: ops.int8_gemm(x, xs, w, ws, bias, out=got)) == route
    assert _gemm_route(lambda: ops.int8_gemm_chunked(x, xs, w, ws, chunk, bias=bias, out=chunks)) == route
    assert _gemm_route(lambda: ops.int8_gemm_gated_residual(x, xs, w, ws, gate, scratch)) == route


@pytest.mark.parametrize("skip", [1, 2])
@pytest.mark.parametrize("m,n,k,route", [(300, 1024, 8192, (128, 1, 2)), (400, 3064, 8208, (256, 2, 2)), (129, 2056, 16400, (256, 2, 4))])
def test_bounded_wait_of_a_shared_tile_stores_nothing(ops, m, n, k, route, skip):
    """One CTA's wait (skip 2: that of the first part of K only) runs out: no CTA of its cluster has the whole sum, so none stores,
    neither a result nor into the residual stream. The status word is raised and the next call is right."""
    g = _gen(m + n + k)
    x = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
    xs, ws = torch.rand(m, device="cuda", generator=g) * 1e-3, torch.rand(n, device="cuda", generator=g) * 1e-3
    gate, res = torch.randn(n, device="cuda", generator=g).bfloat16(), torch.randn((m, n), device="cuda", generator=g).bfloat16()
    out, got_res = torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda"), res.clone()
    assert _gemm_route(lambda: ops.int8_gemm(x, xs, w, ws, out=out)) == route
    torch.cuda.synchronize()
    assert ops.kernel_status() == (0, 0)
    ops.debug_bounded_wait(2_000_000, skip)
    try:
        ops.int8_gemm(x, xs, w, ws, out=out)
        ops.int8_gemm_gated_residual(x, xs, w, ws, gate, got_res)
        torch.cuda.synchronize()
        assert ops.kernel_status() == (1, 0)
    finally:
        ops.debug_bounded_wait(200_000_000, 0)
        ops.kernel_status_clear()
    assert torch.equal(out, torch.full_like(out, 7.0)) and torch.equal(got_res, res)
    ops.int8_gemm(x, xs, w, ws, out=out)
    assert torch.equal(out.view(torch.int16), ops.int8_gemm(x, xs, w, ws, tile=ops.TILE_128x128).view(torch.int16))
    assert ops.kernel_status() == (0, 0)


@pytest.mark.parametrize("tile", [-1, 4, 16, 17, 18])
def test_gemm_tile_values_outside_the_enum_run_whole_tiles(ops, tile):
    """A tile argument names a shape and never a split of K, which with as few K blocks as here would leave CTAs without any:
    every value that the enum does not have runs 128 x 128 tiles."""
    m, n = 200, 264
    for k in (16, 128, 384):
        g = _gen(k)
        x = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
        w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=g)
        xs, ws = torch.rand(m, device="cuda", generator=g) * 1e-3, torch.rand(n, device="cuda", generator=g) * 1e-3
        gate, res = torch.randn(n, device="cuda", generator=g).bfloat16(), torch.randn((m, n), device="cuda", generator=g).bfloat16()
        got, want = [], []
        for t, to in ((tile, got), (ops.TILE_128x128, want)):
            to += [ops.int8_gemm(x, xs, w, ws, tile=t), ops.int8_gemm_chunked(x, xs, w, ws, 88, tile=t), res.clone()]
            ops.int8_gemm_gated_residual(x, xs, w, ws, gate, to[-1], tile=t)
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert ops.kernel_status() == (0, 0)


@pytest.mark.parametrize("lens", [[1], [33], [64], [65], [297], [512], [320, 266], [17, 0, 512], [100, 448, 3, 64, 449]])
def test_prepass_of_short_sequences_in_one_launch(ops, lens):
    """max_seqlen up to 512: the pre-pass is one launch. The same call with a larger max_seqlen takes the separate kernels."""
    heads, total, batch = 3, sum(lens), len(lens)
    qkv = torch.randn((total, 3 * heads * 128), device="cuda", generator=_gen(total)).bfloat16()
    norms = [(1 + 0.1 * torch.randn(128, device="cuda", generator=_gen(i))).bfloat16() for i in (1, 2)]
    table = torch.cat([ops.moss_rope_table(1, 1, n - 1) for n in lens if n > 0]).contiguous()
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    got = []
    for longest in (max(lens), 1025):
        x = qkv.clone()
        q, k, v = (x[:, i * heads * 128:(i + 1) * heads * 128].unflatten(1, (heads, 128)) for i in range(3))
        l = ops.attention_q8_layout(total, total, batch, longest, heads)
        ws = torch.full((l.total,), 0x55, dtype=torch.uint8, device="cuda")
        ops.attention_q8_preprocess(q, k, v, cu, cu, longest, workspace=ws, norm_rope=(norms[0], norms[1], table))
        cut = lambda at, *shape: ws[at:at + int(np.prod(shape))].view(*shape).clone()
        rows = [cut(at, total * heads, 128) for at in (l.q_i8, l.k_i8, l.v8)]
        stats = [cut(at, batch * heads, 512) for at in (l.k_mean, l.v_scale, l.v_recp)]
        qs, ks = cut(l.q_scale, batch * heads, 4 * l.q_blocks), cut(l.k_scale, batch * heads, 4 * l.k_blocks)
        n = (max(lens) + 127) // 128 * 16, (max(lens) + 63) // 64 * 4
        got.append([x.view(torch.int16), *rows, *stats, qs[:, :n[0]], ks[:, :n[1]]])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens", [[1], [297], [17, 0, 512], [100, 448, 3, 64, 449]])
def test_prepass_in_one_launch_leaves_the_whole_layout(ops, lens):
    """Every area of the documented workspace layout that the separate kernels fill: the partial sums and maxima too, which with
    sequences of one chunk are the channel's sum and maximum."""
    heads, total, batch = 3, sum(lens), len(lens)
    qkv = torch.randn((total, 3 * heads * 128), device="cuda", generator=_gen(total)).bfloat16()
    norm, table = torch.ones(128, dtype=torch.bfloat16, device="cuda"), ops.moss_rope_table(1, 1, total - 1)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    got = []
    for longest in (max(lens), 513):  # one launch; the separate kernels, whose second chunk is empty
        q, k, v = (qkv.clone()[:, i * heads * 128:(i + 1) * heads * 128].unflatten(1, (heads, 128)) for i in range(3))
        l = ops.attention_q8_layout(total, total, batch, longest, heads)
        ws = torch.full((l.total,), 0x55, dtype=torch.uint8, device="cuda")
        call = lambda: ops.attention_q8_preprocess(q, k, v, cu, cu, longest, workspace=ws, norm_rope=(norm, norm, table))
        assert len(_kernels(call)) == (1 if longest <= 512 else 4)
        q, k, v = (qkv.clone()[:, i * heads * 128:(i + 1) * heads * 128].unflatten(1, (heads, 128)) for i in range(3))
        call()
        parts = [ws[at:at + batch * heads * l.chunks * 512].view(torch.int32).view(batch, heads, l.chunks, 128)[:, :, 0].clone()
                 for at in (l.part_sum, l.part_amax)]
        assert l.chunks == (1 if longest <= 512 else 2)
        got.append(parts)
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("layout", ["apart", "heads first", "padded rows", "head gaps"])
def test_prepass_in_one_launch_for_other_strides(ops, layout):
    """q, k and v in tensors of their own, with the heads outermost, with rows or heads that leave a gap, a table whose rows leave
    one, and values in another layout than the keys: one launch and the separate kernels give the same."""
    heads, lens = 4, [65, 0, 300, 1]
    total, batch = sum(lens), len(lens)
    shape = {"apart": (total, heads, 128), "heads first": (heads, total, 128), "padded rows": (total, heads * 128 + 40), "head gaps": (total, heads, 136)}[layout]
    view = {"apart": lambda t: t, "heads first": lambda t: t.transpose(0, 1), "padded rows": lambda t: t[:, :heads * 128].unflatten(1, (heads, 128)),
            "head gaps": lambda t: t[:, :, :128]}[layout]
    norms = [(1 + 0.1 * torch.randn(128, device="cuda", generator=_gen(i))).bfloat16() for i in (1, 2)]
    table = torch.cat([ops.moss_rope_table(1, 1, n - 1) for n in lens if n > 0])
    wide = torch.zeros((total, table.shape[1] + 64), dtype=torch.bfloat16, device="cuda")
    wide[:, :table.shape[1]] = table
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    got = []
    for longest in (300, 513):
        tq, tk = (torch.randn(shape, device="cuda", generator=_gen(i)).bfloat16() for i in (3, 4))
        q, k, v = view(tq), view(tk), torch.randn((heads, total, 128), device="cuda", generator=_gen(5)).bfloat16().transpose(0, 1)
        l = ops.attention_q8_layout(total, total, batch, longest, heads)
        ws = torch.full((l.total,), 0x55, dtype=torch.uint8, device="cuda")
        call = lambda: ops.attention_q8_preprocess(q, k, v, cu, cu, longest, workspace=ws, norm_rope=(norms[0], norms[1], wide[:, :table.shape[1]]))
        assert len(_kernels(call)) == (1 if longest <= 512 else 4)
        call()
        cut = lambda at, *shape: ws[at:at + int(np.prod(shape))].view(*shape).clone()
        scales = [cut(at, batch * heads, 4 * n)[:, :4 * m] for at, n, m in ((l.q_scale, l.q_blocks, 12), (l.k_scale, l.k_blocks, 5))]
        got.append([tk.view(torch.int16), *(cut(at, total * heads, 128) for at in (l.q_i8, l.k_i8, l.v8)),
                    *(cut(at, batch * heads, 512) for at in (l.k_mean, l.v_scale, l.v_recp)), *scales])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("heads,lens,longest,one", [(3, [20], 512, True), (24, [297, 290], 297, True), (24, [494, 489], 504, True),
                                                    (24, [20], 512, False), (24, [20, 20], 512, False), (12, [140, 130], 512, False),
                                                    (24, [512] * 3, 512, False), (4, [100] * 32, 512, False), (1, [7] * 60, 512, False)])
def test_prepass_in_one_launch_only_where_it_is_the_faster(ops, heads, lens, longest, one):
    """A CTA for every 64 rows up to max_seqlen: many sequences, or a max_seqlen far above their lengths, take the separate
    kernels, which look at an empty block once and leave."""
    total = sum(lens)
    qkv = torch.randn((total, 3 * heads * 128), device="cuda", generator=_gen(total)).bfloat16()
    q, k, v = (qkv[:, i * heads * 128:(i + 1) * heads * 128].unflatten(1, (heads, 128)) for i in range(3))
    norm = torch.ones(128, device="cuda").bfloat16()
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    ws = torch.empty(ops.attention_q8_workspace_bytes(total, total, len(lens), longest, heads), dtype=torch.uint8, device="cuda")
    table = ops.moss_rope_table(1, 1, total - 1)
    names = _kernels(lambda: ops.attention_q8_preprocess(q, k, v, cu, cu, longest, workspace=ws, norm_rope=(norm, norm, table)))
    assert len(names) == (1 if one else 4), names


@pytest.mark.parametrize("lens,keys", [([300, 64, 700, 129], None), ([1, 0, 257, 40], [513, 70, 64, 900]), ([130] + [40] * 31, None), ([200] + [33] * 33, None)])
def test_attention_of_a_batch_is_that_of_its_sequences(ops, lens, keys):
    """Sequences of different lengths are handed out longest first up to 32 of them, in batch order beyond."""
    heads, keys = 2, keys or lens
    q = torch.randn((sum(lens), heads, 128), device="cuda", generator=_gen(5)).bfloat16()
    k, v = (torch.randn((sum(keys), heads, 128), device="cuda", generator=_gen(s)).bfloat16() for s in (6, 7))
    cu = lambda n: torch.tensor(np.concatenate([[0], np.cumsum(n)]), dtype=torch.int32, device="cuda")
    out, want = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
    ops.attention_q8(q, k, v, out, cu(lens), cu(keys), max(lens + keys), ops.SM_SCALE)
    a = b = 0
    for n, m in zip(lens, keys):
        if n > 0:
            ops.attention_q8(q[a:a + n], k[b:b + m], v[b:b + m], want[a:a + n], cu([n]), cu([m]), max(n, m), ops.SM_SCALE)
        a, b = a + n, b + m
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert ops.kernel_status() == (0, 0)


@pytest.mark.parametrize("heads,lens,keys,longest,by_length", [
    (64, [300, 64, 700, 129], None, 700, True), (64, [1, 0, 257, 40], [513, 70, 64, 900], 900, True), (12, [130] + [40] * 31, None, 130, True),
    (12, [129] * 31, None, 16384, True), (64, [128, 1, 129, 1], None, 5000, True), (64, [1] * 32, None, 512, True), (64, [0, 128, 0, 513], None, 513, True),
    (64, [200] + [33] * 33, None, 200, False), (7, [300, 64, 700, 129], None, 700, True), (3, [130, 2], None, 4096, True), (64, [300, 290], None, 300, False),
    (3, [300, 64, 700, 129], None, 700, False), (1, [130, 2], None, 4096, False)])
def test_attention_by_length_reaches_every_tile(ops, heads, lens, keys, longest, by_length):
    """Sequences of different lengths are handed out longest first, up to 32 of them and where batch order has more CTAs than there
    are SMs; else in batch order. The flat grid has to
    reach the last tile whatever the lengths leave of each tile."""
    keys = keys or lens
    q = torch.randn((sum(lens), heads, 128), device="cuda", generator=_gen(5)).bfloat16()
    k, v = (torch.randn((sum(keys), heads, 128), device="cuda", generator=_gen(s)).bfloat16() for s in (6, 7))
    cu = lambda n: torch.tensor(np.concatenate([[0], np.cumsum(n)]), dtype=torch.int32, device="cuda")
    out, want, cq, ck = torch.full_like(q, 7.0), torch.full_like(q, 7.0), cu(lens), cu(keys)
    ws = torch.empty(ops.attention_q8_workspace_bytes(sum(lens), sum(keys), len(lens), longest, heads), dtype=torch.uint8, device="cuda")
    call = lambda: ops.attention_q8(q, k, v, out, cq, ck, longest, ops.SM_SCALE, workspace=ws)
    call()
    a = b = 0
    for n, m in zip(lens, keys):
        if n > 0:
            ops.attention_q8(q[a:a + n], k[b:b + m], v[b:b + m], want[a:a + n], cu([n]), cu([m]), max(n, m), ops.SM_SCALE)
        a, b = a + n, b + m
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert ops.kernel_status() == (0, 0)
    assert ("ILb0ELb1E" in _kernels(call)[-1]) == by_length, _kernels(call)[-1]


@pytest.mark.parametrize("lens", [[129], [4160], [8192, 1, 3000]])
def test_attention_does_not_depend_on_what_shares_the_sms(ops, lens):
    """P lies where later scores go: a head's output is the same bits with two CTAs on an SM, alone, and in every one of many
    launches (short and long pipelines, scores that make the softmax raise its reference)."""
    heads, total = 24, sum(lens)
    q, k, v = (torch.randn((total, heads, 128), device="cuda", generator=_gen(s)) for s in (8, 9, 10))
    k = (k * torch.linspace(0.1, 5.0, total, device="cuda")[:, None, None]).bfloat16()
    q, v = q.bfloat16(), v.bfloat16()
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    out, first = torch.empty_like(q), torch.empty_like(q)
    ws = torch.empty(ops.attention_q8_workspace_bytes(total, total, len(lens), max(lens), heads), dtype=torch.uint8, device="cuda")
    ops.attention_q8(q, k, v, first, cu, cu, max(lens), ops.SM_SCALE, workspace=ws)
    for _ in range(20):
        ops.attention_q8(q, k, v, out.fill_(7.0), cu, cu, max(lens), ops.SM_SCALE, workspace=ws)
        assert torch.equal(out.view(torch.int16), first.view(torch.int16))
    for h in (0, 11, 23):
        one = out[:, h:h + 1].clone()
        ops.attention_q8(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], one, cu, cu, max(lens), ops.SM_SCALE)
        assert torch.equal(one.view(torch.int16), first[:, h:h + 1].view(torch.int16))
    assert ops.kernel_status() == (0, 0)

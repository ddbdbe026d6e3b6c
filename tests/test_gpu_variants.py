"""Kernel variants chosen by size, alignment or option, each at the sizes where its choice or its edges lie, held to the
CPU oracle or to the bits of the form it stands in for."""
import numpy as np
import pytest
import torch

from oracle import oracle_lib as orc
from owoinfer_b200 import synth

pytestmark = pytest.mark.gpu
D, H = 3072, 24


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from owoinfer_b200 import ops as o
    yield o
    torch.cuda.synchronize()
    assert o.kernel_status() == (0, 0)


def bits(t):
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


# An item is 16 columns; a block takes 1024 of them at a time, the grid at most 8 blocks per SM. Two items; remainders of a
# block's step; just under one step of the whole grid (148 SMs: 1212416 items), and a second step with a remainder.
@pytest.mark.parametrize("rows,k,group", [(1, 32, 16), (3, 96, 32), (37, 3072, 64), (5, 3072, 48), (1300, 12288, 128), (1603, 12288, 128)])
def test_four_bit_weights_to_int8(ops, rows, k, group):
    rng = np.random.default_rng(rows)
    packed = rng.integers(0, 256, (rows, k // 2), dtype=np.uint8)
    dp = torch.from_numpy(packed).cuda()
    assert np.array_equal(ops.unpack_int4(dp).cpu().numpy(), orc.unpack_int4(packed))
    if (rows, k) == (1603, 12288):
        assert 1024 * 8 * torch.cuda.get_device_properties(0).multi_processor_count < rows * k // 16
    if rows > 1:  # padded rows on both sides
        wide, out = torch.zeros((rows, k // 2 + 16), dtype=torch.uint8, device="cuda"), torch.full((rows, k + 16), 99, dtype=torch.int8, device="cuda")
        wide[:, :k // 2] = dp
        ops.unpack_int4(wide[:, :k // 2], out=out[:, :k])
        assert np.array_equal(out[:, :k].cpu().numpy(), orc.unpack_int4(packed)) and (out[:, k:] == 99).all()
    e4m3 = rng.integers(0x18, 0x58, (rows, k // group), dtype=np.uint8)
    fp16 = (rng.random((rows, k // group)).astype(np.float32) * 12 + 0.01).astype(np.float16).view(np.uint16)
    cb = rng.normal(0, 4, 16).astype(np.float32)
    for scales, dev in ((e4m3, torch.from_numpy(e4m3).cuda()), (fp16, torch.from_numpy(fp16.view(np.int16)).cuda())):
        want = orc.decode_grouped_int8(packed, scales, group)
        assert np.array_equal(ops.decode_grouped_int8(dp, dev, group).cpu().numpy(), want)
        want = orc.decode_grouped_int8(packed, scales, group, cb)
        assert np.array_equal(ops.decode_grouped_int8(dp, dev, group, torch.from_numpy(cb).cuda()).cpu().numpy(), want)


@pytest.mark.parametrize("slot,n0,n1", [(7, 65, 1), (128, 200, 333)])
def test_tap_and_slots_read_in_place_equal_the_copied_forms(ops, slot, n0, n1):
    """k | v rows tapped by the pass that quantises them, and slot rows read where they lie, against the copies that rows
    without 16-byte alignment take, and against the separate QK-norm + RoPE."""
    F = 512
    w = synth.block_weights(D, F, 31)
    bw = ops.BlockWeights(w["norm1"], w["norm2"], w["q_norm"], w["k_norm"], w["qkv"], w["o"], w["up_gate"], w["down"])
    mod, L = synth.modulation(D, 4), n0 + n1
    x0 = synth.activations(L, D, 9)
    rope = ops.moss_rope_table(1, 1, L - 1)
    cu = synth.cu_seqlens([n0, n1])

    def run(**kw):
        r = ops.block_run(L, cu, max(n0, n1) + kw.pop("extra", 0), D=D, F=F, **kw)
        ws = torch.empty(ops.block_quant_workspace_bytes(r), dtype=torch.uint8, device="cuda")
        x = x0.clone()
        ops.run_block_quant(bw, ops.block_buffers(x, mod, rope, ws), r)
        torch.cuda.synchronize()
        return bits(x)

    flat = torch.zeros(L * 2 * D + 8, dtype=torch.bfloat16, device="cuda")
    taps = [flat[o:o + L * 2 * D].view(L, 2 * D) for o in (0, 4)]      # the second one only 8-byte aligned
    seen = []
    for tap in taps:
        tap.zero_()
        seen.append((run(kv_tap=tap), bits(tap)))
    plain = run()
    assert all(np.array_equal(y, plain) for y, _ in seen) and np.array_equal(seen[0][1], seen[1][1]) and seen[0][1].any()

    kv = torch.randn(slot * 2 * D + 8, device="cuda", generator=torch.Generator("cuda").manual_seed(slot)).to(torch.bfloat16)
    odd = torch.empty_like(kv)
    odd[4:4 + slot * 2 * D] = kv[:slot * 2 * D]
    aligned, shifted = kv[:slot * 2 * D].view(slot, 2 * D), odd[4:4 + slot * 2 * D].view(slot, 2 * D)
    both = dict(slot_rows=slot, cu_seqlens_k=synth.cu_seqlens([slot + n0, n1 + slot]), k0=0, k1=L + 2 * slot, extra=slot)
    want = run(slot_kv=(shifted, shifted), **both)
    assert np.array_equal(run(slot_kv=(aligned, aligned), **both), want)
    assert np.array_equal(run(slot_kv=(aligned, aligned), fused_norm_rope=0, **both), want)
    one = dict(slot_rows=slot, cu_seqlens_k=synth.cu_seqlens([n0, n1 + slot]), k0=slot, k1=L + 2 * slot, extra=slot)
    assert np.array_equal(run(slot_kv=(None, aligned), **one), run(slot_kv=(None, shifted), **one))


@pytest.mark.parametrize("rows", [33, 512, 513])   # the tensor-core kernels let their successor start early up to 512 rows
def test_overlapping_launches_change_no_bit(ops, rows):
    """A step of several blocks, whose launches overlap, against its blocks one by one with a synchronisation after each."""
    F = 512
    ws = [synth.block_weights(D, F, 50 + i) for i in range(3)]
    bws = [ops.BlockWeights(w["norm1"], w["norm2"], w["q_norm"], w["k_norm"], w["qkv"], w["o"], w["up_gate"], w["down"]) for w in ws]
    mod, rope, x0 = synth.modulation(D, 4), ops.moss_rope_table(1, 1, rows - 1), synth.activations(rows, D, 9)
    run = ops.block_run(rows, synth.cu_seqlens([rows]), rows, D=D, F=F)
    work = torch.empty(ops.block_quant_workspace_bytes(run), dtype=torch.uint8, device="cuda")
    one, many = x0.clone(), [x0.clone() for _ in range(4)]
    torch.cuda.synchronize()
    for b in bws:
        ops.run_block_quant(b, ops.block_buffers(one, mod, rope, work), run)
        torch.cuda.synchronize()
    for x in many:
        ops.dit_step(bws, ops.block_buffers(x, mod, rope, work), run)
    torch.cuda.synchronize()
    for x in many:
        assert torch.equal(x.view(torch.int16), one.view(torch.int16))


# Row counts on both sides of where the automatic choice changes: 128 x 128 tiles, 128 x 256 tiles, CTA pairs.
@pytest.mark.parametrize("rows", [1, 128, 129, 256, 257, 385, 737, 769, 1281])
def test_automatic_tile_gives_the_bits_of_every_tile(ops, rows):
    g = torch.Generator("cuda").manual_seed(rows)
    ints = lambda *s: torch.randint(-127, 128, s, dtype=torch.int8, device="cuda", generator=g)
    for n, k in ((9216, 256), (1024, 3072)):
        x, w = ints(rows, k), ints(n, k)
        xs, ws = (torch.rand(s, device="cuda", generator=g) * 1e-3 for s in (rows, n))
        gate, res = (torch.randn(s, device="cuda", generator=g).to(torch.bfloat16) for s in ((n,), (rows, n)))
        forms = (lambda t: ops.int8_gemm(x, xs, w, ws, tile=t), lambda t: ops.int8_gemm_situ_glu(x, xs, w, ws, tile=t),
                 lambda t: ops.int8_gemm_gated_residual(x, xs, w, ws, gate, res.clone(), tile=t))
        for form in forms:
            want = form(ops.TILE_AUTO).view(torch.int16)
            for tile in (ops.TILE_128x128, ops.TILE_128x256, ops.TILE_2CTA_256x256):
                assert torch.equal(form(tile).view(torch.int16), want)
        acc = ops.int8_gemm_acc(x, w)
        rows_ref = slice(0, min(rows, 8))
        assert torch.equal(acc[rows_ref].double(), x[rows_ref].double() @ w.double().T)


def test_rows_outside_the_sequences_are_tapped_and_read_as_keys(ops):
    """cu_seqlens need not cover every row of a run. The tap still holds all rows, and key sequences of a run with slots may
    reach rows that no query sequence covers: the same bits as with the separate QK-norm + RoPE and the copies."""
    F, L, slot, lens = 512, 300, 70, [150, 87]
    w = synth.block_weights(D, F, 31)
    bw = ops.BlockWeights(w["norm1"], w["norm2"], w["q_norm"], w["k_norm"], w["qkv"], w["o"], w["up_gate"], w["down"])
    mod, x0, rope = synth.modulation(D, 4), synth.activations(L, D, 9), ops.moss_rope_table(1, 1, L - 1)
    cu = (synth.cu_seqlens(lens) + 13).contiguous()                      # rows 0..12 and 250..299 lie outside
    inside = slice(13, 13 + sum(lens))

    def run(max_len, **kw):
        r = ops.block_run(L, cu, max_len, D=D, F=F, **kw)
        ws = torch.zeros(ops.block_quant_workspace_bytes(r), dtype=torch.uint8, device="cuda")
        x = x0.clone()
        ops.run_block_quant(bw, ops.block_buffers(x, mod, rope, ws), r)
        torch.cuda.synchronize()
        return bits(x[inside])

    xq, xs = ops.rotate_quantize(ops.rms_norm_modulate(x0, w["norm1"], mod[D:2 * D], mod[:D]))
    qkv = ops.int8_gemm(xq, xs, w["qkv"][0], w["qkv"][1])
    ops.qk_norm_rope_moss(qkv, H, w["q_norm"], w["k_norm"], rope)
    plain = run(150)
    for fused in (-1, 0):
        tap = torch.zeros((L, 2 * D), dtype=torch.bfloat16, device="cuda")
        assert np.array_equal(run(150, kv_tap=tap, fused_norm_rope=fused), plain)
        assert np.array_equal(bits(tap), bits(qkv[:, D:]))

    kv = torch.randn(slot * 2 * D + 8, device="cuda", generator=torch.Generator("cuda").manual_seed(7)).to(torch.bfloat16)
    odd = torch.empty_like(kv)
    odd[4:4 + slot * 2 * D] = kv[:slot * 2 * D]                          # only 8-byte aligned: the copies
    aligned, shifted = kv[:slot * 2 * D].view(slot, 2 * D), odd[4:4 + slot * 2 * D].view(slot, 2 * D)
    # Keys of the first sequence: slot A and own rows 0..162; of the second: own rows 163..299 and slot B.
    both = dict(slot_rows=slot, cu_seqlens_k=synth.cu_seqlens([slot + 163, L - 163 + slot]), k0=0, k1=L + 2 * slot)
    want = run(slot + 163, slot_kv=(shifted, shifted), **both)
    assert np.array_equal(run(slot + 163, slot_kv=(aligned, aligned), **both), want)
    assert np.array_equal(run(slot + 163, slot_kv=(aligned, aligned), fused_norm_rope=0, **both), want)
    own = dict(slot_rows=slot, cu_seqlens_k=synth.cu_seqlens([163, L - 163]), k0=slot, k1=slot + L)   # neither slot read
    assert np.array_equal(run(163, slot_kv=(None, None), **own), run(163, slot_kv=(None, None), fused_norm_rope=0, **own))


def test_key_rows_past_the_last_sequence_do_not_reach_the_output(ops):
    """The last key tile of the last sequence may hold rows that no sequence covers; whatever the workspace holds there
    (here NaN bytes) has no part in the output."""
    lens, extra = [70, 200], 61
    total = sum(lens)
    g = torch.Generator("cuda").manual_seed(3)
    q = torch.randn((total, 2, 128), device="cuda", generator=g).to(torch.bfloat16)
    k, v = (torch.randn((total + extra, 2, 128), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    cu, outs = synth.cu_seqlens(lens), []
    for rows in (total, total + 1, total + extra):
        ws = torch.full((ops.attention_q8_workspace_bytes(total, rows, 2, 200, 2),), 0x7f, dtype=torch.uint8, device="cuda")
        out = torch.zeros_like(q)
        ops.attention_q8(q, k[:rows], v[:rows], out, cu, cu, 200, ops.SM_SCALE, workspace=ws)
        torch.cuda.synchronize()
        outs.append(bits(out))
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


class Serial:
    """A block call by call through the separate public ops, synchronised after each: no launch overlaps another one's
    call. (The launches inside one attention call still overlap; those are held to the oracle elsewhere.)"""

    def __init__(self, ops, tier, w, F):
        self.o, self.tier, self.w, self.F = ops, tier, w, F
        self.packed = {n: ops.make_w4(w[n][0], w[n][1], 64, w[n][2]) if tier == ops.TIER_W4A8 else w[n] for n in ("qkv", "o", "up_gate", "down")}
        self.block = ops.BlockWeights(w["norm1"], w["norm2"], w["q_norm"], w["k_norm"], *self.packed.values())

    def do(self, f, *a, **kw):
        out = f(*a, **kw)
        torch.cuda.synchronize()
        return out

    def quant(self, x, *norm):
        if self.tier != self.o.TIER_W4A4_VIA_INT8:
            return self.do(self.o.rms_norm_modulate_rotate_quantize if norm else self.o.rotate_quantize, x, *norm)
        q, s = self.do(self.o.rms_norm_modulate_convrot_quantize_int4 if norm else self.o.convrot_quantize_int4, x, *norm)
        return self.do(self.o.unpack_int4, q), s

    def site(self, name, xq, xs, epilogue, gate=None, res=None):
        o, lin = self.o, self.packed[name]
        if self.tier == o.TIER_W4A8:
            return self.do(o.w4a8_gemm, xq, xs, lin, self.w[name][0].shape[0], epilogue, gate, res)
        w, s = (lin[0] if self.tier == o.TIER_INT8 else self.do(o.unpack_int4, lin[0])), lin[1]
        if epilogue == 1:
            return self.do(o.int8_gemm_gated_residual, xq, xs, w, s, gate, res)
        return self.do(o.int8_gemm if epilogue == 0 else o.int8_gemm_situ_glu, xq, xs, w, s)

    def __call__(self, x, mod, rope, cu, max_len, slots=None, cu_k=None):
        """x in place; slots: (slot A, slot B) rows k | v. Returns the k | v rows of the run (the tap)."""
        o, w, m, L = self.o, self.w, [mod[i * D:(i + 1) * D] for i in range(6)], x.shape[0]
        qkv = self.site("qkv", *self.quant(x, w["norm1"], m[1], m[0]), 0)
        self.do(o.qk_norm_rope_moss, qkv, H, w["q_norm"], w["k_norm"], rope)
        kv = qkv[:, D:]
        if slots is not None:
            kv = torch.cat([slots[0], kv, slots[1]])
        heads = lambda t, at: t.as_strided((t.shape[0], H, 128), (t.stride(0), 128, 1), t.storage_offset() + at)
        attn = torch.empty((L, D), dtype=torch.bfloat16, device="cuda")
        self.do(o.attention_q8, heads(qkv, 0), heads(kv, 0), heads(kv, D), attn.view(L, H, 128), cu, cu if cu_k is None else cu_k, max_len, o.SM_SCALE)
        self.site("o", *self.quant(attn), 1, m[2], x)
        ffn = self.site("up_gate", *self.quant(x, w["norm2"], m[4], m[3]), 2)
        self.site("down", *self.quant(ffn), 1, m[5], x)
        return qkv[:, D:].contiguous()


@pytest.fixture(scope="module")
def serial_blocks(ops):
    F = 1024
    return {t: [Serial(ops, t, synth.block_weights(D, F, 70 + 10 * i, tier=t), F) for i in range(2)]
            for t in (ops.TIER_INT8, ops.TIER_W4A4_VIA_INT8, ops.TIER_W4A8)}


@pytest.mark.parametrize("tier", [0, 1, 2])
@pytest.mark.parametrize("rows", [33, 512, 513])   # the tensor-core kernels let their successor start early up to 512 rows
def test_a_step_of_overlapping_launches_equals_its_calls_one_by_one(ops, serial_blocks, tier, rows):
    """Two blocks in one chain of launches, eagerly and replayed from a graph, against every call by itself."""
    blocks = serial_blocks[tier]
    lens = [rows - rows // 3, rows // 3]
    mod, rope, x0 = synth.modulation(D, 4), ops.moss_rope_table(1, 1, rows - 1), synth.activations(rows, D, 9)
    cu = synth.cu_seqlens(lens)
    want = x0.clone()
    for b in blocks:
        b(want, mod, rope, cu, lens[0])
    run = ops.block_run(rows, cu, lens[0], D=D, F=blocks[0].F, tier=tier)
    work = torch.empty(ops.block_quant_workspace_bytes(run), dtype=torch.uint8, device="cuda")
    x = x0.clone()
    step = lambda: ops.dit_step([b.block for b in blocks], ops.block_buffers(x, mod, rope, work), run)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for go in (step, graph.replay):
        for _ in range(4):
            work.fill_(0x7f)                        # a value read before it is written shows
            x.copy_(x0)
            go()
            torch.cuda.synchronize()
            assert torch.equal(x.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("tier", [0, 1, 2])
@pytest.mark.parametrize("n0,n1", [(20, 13), (300, 333)])
def test_taps_and_slots_in_a_chain_equal_the_calls_one_by_one(ops, serial_blocks, tier, n0, n1):
    b, slot, L = serial_blocks[tier][0], 65, n0 + n1
    mod, rope, x0 = synth.modulation(D, 4), ops.moss_rope_table(1, 1, L - 1), synth.activations(L, D, 9)
    cu, kv = synth.cu_seqlens([n0, n1]), torch.randn((2, slot, 2 * D), device="cuda", generator=torch.Generator("cuda").manual_seed(n0)).to(torch.bfloat16)

    def chain(**kw):
        r = ops.block_run(L, cu, max(n0, n1) + slot, D=D, F=b.F, tier=tier, **kw)
        x, work = x0.clone(), torch.full((ops.block_quant_workspace_bytes(r),), 0x7f, dtype=torch.uint8, device="cuda")
        ops.run_block_quant(b.block, ops.block_buffers(x, mod, rope, work), r)
        torch.cuda.synchronize()
        return bits(x)

    want, tap = x0.clone(), torch.zeros((L, 2 * D), dtype=torch.bfloat16, device="cuda")
    rows = b(want, mod, rope, cu, max(n0, n1) + slot)
    assert np.array_equal(chain(kv_tap=tap), bits(want)) and np.array_equal(bits(tap), bits(rows))
    # Both slots; then key rows that begin (and end) inside the run's own rows, which keep the copies.
    want, cu_k = x0.clone(), synth.cu_seqlens([slot + n0, n1 + slot])
    b(want, mod, rope, cu, max(n0, n1) + slot, slots=kv, cu_k=cu_k)
    assert np.array_equal(chain(slot_rows=slot, slot_kv=(kv[0], kv[1]), cu_seqlens_k=cu_k, k0=0, k1=L + 2 * slot), bits(want))
    want, cut = x0.clone(), 5
    b(want, mod, rope, cu, max(n0, n1) + slot, slots=(kv[0], kv[1]), cu_k=synth.cu_seqlens([n0 - cut, n1 + slot]) + slot + cut)
    got = chain(slot_rows=slot, slot_kv=(None, kv[1]), cu_seqlens_k=synth.cu_seqlens([n0 - cut, n1 + slot]), k0=slot + cut, k1=L + 2 * slot)
    assert np.array_equal(got, bits(want))
    want = x0.clone()
    b(want, mod, rope, cu, max(n0, n1) + slot, slots=(kv[0], kv[1]), cu_k=synth.cu_seqlens([slot + n0, n1 - cut]))
    got = chain(slot_rows=slot, slot_kv=(kv[0], None), cu_seqlens_k=synth.cu_seqlens([slot + n0, n1 - cut]), k0=0, k1=slot + L - cut)
    assert np.array_equal(got, bits(want))

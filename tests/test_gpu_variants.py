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


# One item; a remainder of the 1024-item step of a block; more items than one step of the whole grid takes.
@pytest.mark.parametrize("rows,k,group", [(1, 32, 16), (3, 96, 32), (37, 3072, 64), (5, 3072, 48), (1300, 12288, 128)])
def test_four_bit_weights_to_int8(ops, rows, k, group):
    rng = np.random.default_rng(rows)
    packed = rng.integers(0, 256, (rows, k // 2), dtype=np.uint8)
    dp = torch.from_numpy(packed).cuda()
    assert np.array_equal(ops.unpack_int4(dp).cpu().numpy(), orc.unpack_int4(packed))
    if k % 32 == 0 and rows > 1:  # padded rows on both sides
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

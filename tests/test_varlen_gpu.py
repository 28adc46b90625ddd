"""GPU: streaming attention over a packed batch (``cu_seqlens``), an extension of the reference's operator.

The packed call must equal the padded call (``streaming_attention`` with ``lens``) row for row and bit for
bit: both run the same tcgen05 kernels over the same tiles of every sequence, the packed one in one launch per
kernel over the whole batch or, with ``single_launch=False``, through strided views of the packed tensors.  The padded call in turn is pinned to the oracle by the other GPU tests; one case
here is also checked against the oracle directly, per sequence, with the benchmark contract's tolerances.
"""

import pytest
import torch

from kernels_b200 import _lib
from oracle import streaming_attention_oracle as SO

pytestmark = pytest.mark.gpu


def _pack(t, lens):
    """[B, H, T, D] padded -> [total, H, D] packed."""
    return torch.cat([t[b, :, :L].transpose(0, 1) for b, L in enumerate(lens)], dim=0).contiguous()


def _cu(lens):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)


@pytest.mark.parametrize("H,Hk,T,D,c,back,dtype,lens", [
    (4, 4, 700, 128, 48, 3, torch.bfloat16, [700, 333, 1]),
    (8, 2, 520, 64, 128, 1, torch.float16, [130, 520, 0, 257]),   # shared K/V heads, an empty sequence
    (2, 2, 1100, 128, 256, 2, torch.float16, [1100, 1024]),
    (3, 1, 300, 64, 10, 5, torch.bfloat16, [299, 17, 128]),
    (2, 2, 260, 128, 32, 2, torch.float16, [5, 130, 256, 257, 1, 127, 128, 129, 0, 260]),  # every kind of last tile
    (8, 8, 2600, 128, 64, 2, torch.bfloat16, [2600, 130, 2500]),  # more tiles per sequence than CTAs: a CTA's next
    (8, 8, 2600, 64, 100, 1, torch.float16, [130, 2600, 2571]),   # item is of the same sequence
    # the same in the long-item class (head dim 128, chunks of 128 rows or more), first of a sequence between others
    (8, 8, 2600, 128, 256, 2, torch.bfloat16, [130, 2600, 2500]),
    (8, 8, 2600, 128, 130, 3, torch.float16, [2571, 2600, 1]),
    # ... and with shared key/value heads: more (key tile, key/value head) items per sequence than CTAs too
    (16, 8, 2600, 128, 256, 2, torch.bfloat16, [2500, 77, 2600]),
    (16, 8, 2600, 64, 64, 2, torch.float16, [300, 2600, 2500]),
    # few tiles per sequence, more items than CTAs
    (4, 4, 500, 64, 10, 4, torch.float16, [(37 * i) % 501 for i in range(60)]),
    (4, 2, 1000, 128, 64, 2, torch.bfloat16, [(61 * i) % 1001 for i in range(40)]),
    # one long sequence among short ones: the grid has a block per tile of the batch and not of the longest sequence;
    # more sequences than a warp has lanes, than it has lanes squared; and lengths for which it stays as it is
    (2, 2, 1500, 128, 64, 2, torch.bfloat16, [1, 0, 128, 129, 256, 257, 0, 1500] + [3] * 40 + [255]),
    (2, 1, 900, 64, 10, 4, torch.float16, [5] * 700 + [900] + [2] * 400),
    (4, 4, 256, 128, 128, 1, torch.bfloat16, [256] * 50),
])
@pytest.mark.parametrize("single_launch", [True, False])
def test_packed_equals_padded_bitwise(H, Hk, T, D, c, back, dtype, lens, single_launch):
    from kernels_b200.streaming_attention import streaming_attention, streaming_attention_varlen

    B = len(lens)
    g = torch.Generator().manual_seed(11)
    q = torch.randn(B, H, T, D, generator=g).to(dtype).cuda()
    k, v = (torch.randn(B, Hk, T, D, generator=g).to(dtype).cuda() for _ in range(2))
    do = torch.randn(B, H, T, D, generator=g).to(dtype).cuda()
    lens_t = torch.tensor(lens, dtype=torch.int32).cuda()
    valid = (torch.arange(T, device="cuda")[None] < lens_t[:, None])[:, None, :, None]
    do = do * valid

    qp, kp, vp = (t.detach().clone().requires_grad_() for t in (q, k, v))
    out_pad, lse_pad = streaming_attention(qp, kp, vp, lens_t, c, back, return_lse=True)
    out_pad.backward(do)

    qs, ks, vs = (_pack(t, lens).requires_grad_() for t in (q, k, v))
    n0 = _lib.launch_count()
    out, lse = streaming_attention_varlen(qs, ks, vs, _cu(lens), c, back, return_lse=True, single_launch=single_launch)
    n1 = _lib.launch_count()
    out.backward(_pack(do, lens))
    torch.cuda.synchronize()
    n2 = _lib.launch_count()
    _lib.check_device_status()
    live = sum(1 for L in lens if L > 0)
    # one launch of each kernel (forward; delta, main, dQ) for the whole batch, or one per sequence
    assert n1 - n0 == (1 if single_launch else live) and n2 - n1 == (3 if single_launch else 3 * live)

    assert out.shape == qs.shape and lse.shape == (H, sum(lens))
    assert torch.equal(out, _pack(out_pad.detach(), lens))
    assert torch.equal(lse, torch.cat([lse_pad[b, :, :L] for b, L in enumerate(lens)], dim=1))
    assert torch.equal(qs.grad, _pack(qp.grad, lens))
    assert torch.equal(ks.grad, _pack(kp.grad, lens))
    assert torch.equal(vs.grad, _pack(vp.grad, lens))


@pytest.mark.parametrize("D,c,back,dtype", [(128, 64, 2, torch.bfloat16), (128, 256, 2, torch.bfloat16), (64, 100, 1, torch.float16)])
def test_more_tiles_per_sequence_than_ctas_against_64_bits(D, c, back, dtype):
    """Padded and packed, ragged, every CTA of the main and the dQ kernel meeting several tiles of one sequence: every
    128-row tile of every head against the 64-bit result (a tile computed with another item's sequence would be off by
    about 1).  Bounds: four times the largest error of a tile measured over 800 random cases (3.3e-3 bf16, 4.3e-4 fp16)."""
    from kernels_b200.streaming_attention import streaming_attention, streaming_attention_varlen

    H, T, lens = 8, 2600, [130, 2600, 2571]
    assert H * -(-T // 128) > torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v, do = (torch.randn(3, H, T, D, generator=g, device="cuda").to(dtype) for _ in range(4))
    chunk = torch.arange(T, device="cuda") // c
    diff = chunk[:, None] - chunk[None]
    mask = (diff >= 0) & (diff <= back)

    padded_in = [t.clone().requires_grad_() for t in (q, k, v)]
    padded = streaming_attention(*padded_in, torch.tensor(lens, dtype=torch.int32, device="cuda"), c, back)
    padded = [padded.detach(), *torch.autograd.grad(padded, padded_in, do)]
    packed_in = [_pack(t, lens).requires_grad_() for t in (q, k, v)]
    packed = streaming_attention_varlen(*packed_in, _cu(lens), c, back)
    packed = [packed.detach(), *torch.autograd.grad(packed, packed_in, _pack(do, lens))]
    bound = {torch.bfloat16: 1.3e-2, torch.float16: 1.8e-3}[dtype]
    r0 = 0
    for b, L in enumerate(lens):
        ref = [t[b, :, :L].double().requires_grad_() for t in (q, k, v)]
        scores = (ref[0] @ ref[1].mT * D**-0.5).masked_fill(~mask[:L, :L], -1e300)
        want = torch.softmax(scores, -1) @ ref[2]
        want = [want.detach(), *torch.autograd.grad(want, ref, do[b, :, :L].double())]
        for name, exact, pad, pack in zip(("o", "dq", "dk", "dv"), want, padded, packed):
            for form, got in (("padded", pad[b, :, :L]), ("packed", pack[r0:r0 + L].transpose(0, 1))):
                for t0 in range(0, L, 128):
                    e, x = exact[:, t0:t0 + 128], got[:, t0:t0 + 128].double()
                    rel = (x - e).norm(dim=(1, 2)) / e.norm(dim=(1, 2))
                    assert float(rel.max()) <= bound, (form, name, b, t0, rel.tolist())
            assert not pad[b, :, L:].any(), name  # padding rows are zeros
        r0 += L


def test_blocks_follow_the_rows_of_a_packed_batch():
    """One long sequence among many short ones costs about what its rows cost, not a block for every tile of the longest
    sequence times every sequence: forward and backward take less than six times as long as the long sequence and the short
    ones packed apart (measured 2.7 times, and 26 with such blocks)."""
    from kernels_b200.streaming_attention import streaming_attention_varlen

    def passes(lens):
        q, k, v, do = (torch.randn(sum(lens), 8, 64, device="cuda", dtype=torch.float16).requires_grad_() for _ in range(4))
        cu = _cu(lens)

        def once():
            torch.autograd.grad(streaming_attention_varlen(q, k, v, cu, 100, 1), (q, k, v), do)

        return once

    def device_us(once):
        times = []
        for i in range(8):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            once()
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return sorted(times)[2]

    both, long, short = (device_us(passes(lens)) for lens in ([32768] + [60] * 2000, [32768], [60] * 2000))
    assert both < 6 * (long + short), (both, long, short)


def test_packed_against_oracle_per_sequence():
    from kernels_b200.streaming_attention import streaming_attention_varlen

    H, D, c, back, dtype, lens = 4, 128, 64, 2, torch.bfloat16, [450, 129, 64]
    g = torch.Generator().manual_seed(3)
    total = sum(lens)
    q, k, v, do = (torch.randn(total, H, D, generator=g).to(dtype) for _ in range(4))
    qs, ks, vs = (t.cuda().requires_grad_() for t in (q, k, v))
    out = streaming_attention_varlen(qs, ks, vs, _cu(lens), c, back)
    out.backward(do.cuda())
    torch.cuda.synchronize()
    _lib.check_device_status()
    r0 = 0
    for L in lens:
        sl = slice(r0, r0 + L)
        qf, kf, vf = (t[sl].transpose(0, 1)[None].float().clone().requires_grad_() for t in (q, k, v))
        ref, _, _ = SO.streaming_attention_oracle(qf, kf, vf, c, back, None)
        ref.backward(do[sl].transpose(0, 1)[None].float())
        got = out[sl].detach().cpu().float().transpose(0, 1)[None]
        assert (got - ref.detach()).abs().max() <= 2e-2  # fp16 / bf16 kernel against the fp32 oracle
        for name, gpu_grad, ref_grad in (("dq", qs.grad, qf.grad), ("dk", ks.grad, kf.grad), ("dv", vs.grad, vf.grad)):
            gg = gpu_grad[sl].cpu().float().transpose(0, 1)[None]
            assert float((gg - ref_grad).norm() / ref_grad.norm()) <= 2e-2, name
        r0 += L


def test_packed_shapes_without_a_tcgen05_kernel_use_the_generic_kernels():
    """fp32 and head dim 32: sequence by sequence through the padded operator (generic CUDA kernels), forward and
    backward, against the oracle per sequence."""
    from kernels_b200.streaming_attention import streaming_attention_varlen

    for dtype, D, tol_o, tol_g in ((torch.float32, 64, 5e-6, 5e-5), (torch.float16, 32, 3e-3, 1e-2)):
        H, c, back, lens = 2, 16, 2, [100, 0, 37]
        g = torch.Generator().manual_seed(4)
        total = sum(lens)
        q, k, v, do = (torch.randn(total, H, D, generator=g).to(dtype) for _ in range(4))
        qs, ks, vs = (t.cuda().requires_grad_() for t in (q, k, v))
        out, lse = streaming_attention_varlen(qs, ks, vs, _cu(lens), c, back, return_lse=True)
        out.backward(do.cuda())
        assert out.shape == q.shape and lse.shape == (H, total)
        r0 = 0
        for L in lens:
            if L == 0:
                continue
            sl = slice(r0, r0 + L)
            qf, kf, vf = (t[sl].transpose(0, 1)[None].float().clone().requires_grad_() for t in (q, k, v))
            ref, _, _ = SO.streaming_attention_oracle(qf, kf, vf, c, back, None)
            ref.backward(do[sl].transpose(0, 1)[None].float())
            assert (out[sl].detach().cpu().float().transpose(0, 1)[None] - ref.detach()).abs().max() <= tol_o
            for gpu_grad, ref_grad in ((qs.grad, qf.grad), (ks.grad, kf.grad), (vs.grad, vf.grad)):
                assert (gpu_grad[sl].cpu().float().transpose(0, 1)[None] - ref_grad).abs().max() <= tol_g
            r0 += L


def test_packed_rejects_bad_offsets():
    from kernels_b200.streaming_attention import streaming_attention_varlen

    q = torch.randn(64, 2, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(AssertionError):
        streaming_attention_varlen(q, q, q, _cu([60]), 16, 1)  # cu_seqlens must end at `total`

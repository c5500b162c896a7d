"""GPU parity: dense attention with LSE (the two-stream dense kernel and the gathering kernel's dense mode, chosen by the number
of waves) against the fp32 oracle.

Tolerances as for the sparse path: max-abs 2e-2, mean-rel 1e-2 on the output; the LSE is fp32 arithmetic
on bf16-rounded products and must agree to 2e-3 absolute."""

import pytest
import torch

from oracle.gather_attn import dense_attn_ref, error_metrics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Lq,Lk,D", [(1000, 1000, 128), (384, 1300, 64), (130, 70, 128), (256, 128, 128), (77, 4000, 128)])
def test_dense_matches_oracle(cuda_device, dtype, Lq, Lk, D):
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention, full_attention_with_lse
    B, H = 2, 3
    g = torch.Generator().manual_seed(Lq * 7 + Lk)
    q = torch.randn(B, H, Lq, D, generator=g).to(dtype)
    k = torch.randn(B, H, Lk, D, generator=g).to(dtype)
    v = torch.randn(B, H, Lk, D, generator=g).to(dtype)
    ref, ref_lse = dense_attn_ref(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2))
    out, lse = full_attention_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
    assert out.shape == q.shape and out.dtype == dtype and lse.shape == (B, H, Lq) and lse.dtype == torch.float32
    mx, mr = error_metrics(out.float().cpu().transpose(1, 2), ref)
    assert mx < 2e-2 and mr < 1e-2, (mx, mr)
    assert float((lse.cpu() - ref_lse).abs().max()) < 2e-3
    out2 = full_attention(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
    assert torch.equal(out2, out)


def test_dense_peaked_rows_and_scale(cuda_device):
    """Rows whose maximum sits in the masked-off part's neighbourhood (last, partial tile) and a custom scale."""
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    B, H, L, D = 1, 2, 300, 128
    g = torch.Generator().manual_seed(3)
    q = torch.randn(B, H, L, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B, H, L, D, generator=g).to(torch.bfloat16)
    k[:, :, -1] = 4 * q[:, :, 0]                      # the very last key dominates row 0
    v = torch.randn(B, H, L, D, generator=g).to(torch.bfloat16)
    ref, ref_lse = dense_attn_ref(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), softmax_scale=0.2)
    out, lse = full_attention_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), scale=0.2)
    mx, mr = error_metrics(out.float().cpu().transpose(1, 2), ref)
    assert mx < 3e-2 and mr < 1e-2, (mx, mr)
    assert float(((lse.cpu() - ref_lse).abs() / ref_lse.abs().clamp_min(1)).max()) < 2e-3


def test_dense_argument_errors(cuda_device):
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention
    q = torch.randn(1, 2, 64, 128, device=cuda_device)
    with pytest.raises(TypeError):
        full_attention(q, q, q)                        # fp32 is not supported
    qh = q.to(torch.bfloat16)
    with pytest.raises(ValueError):
        full_attention(qh, qh[:, :1], qh)              # head count mismatch


# edges of both kernels: one row, one key, stream B empty / one row, several items per CTA; and layouts that no
# tensor map describes (keys shared by all heads: stride 0), which take the gathering kernel
@pytest.mark.parametrize("Lq,Lk,D,shared", [(1, 1, 128, False), (128, 129, 64, False), (129, 127, 128, False), (256, 640, 64, False),
                                            (513, 300, 128, False), (5000, 200, 64, False), (300, 260, 128, True), (257, 130, 64, True),
                                            (5000, 129, 128, False), (1025, 260, 128, False), (1153, 1, 64, False)])
def test_dense_edges(cuda_device, Lq, Lk, D, shared):
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    # (few groups of 128 rows, or five waves of them against three of pairs at D = 128: the gathering kernel; else the other)
    B, H = (1, 18) if Lq >= 1025 else (2, 3)
    g = torch.Generator().manual_seed(Lq + Lk)
    q = torch.randn(B, H, Lq, D, generator=g).to(torch.bfloat16)
    k = (torch.randn(B, 1 if shared else H, Lk, D, generator=g) * torch.linspace(0.2, 3.0, Lk).view(1, 1, Lk, 1)).to(torch.bfloat16)
    v = torch.randn(B, H, Lk, D, generator=g).to(torch.bfloat16)
    perm = torch.stack([torch.randperm(Lq, generator=g) for _ in range(B * H)])
    kd = k.to(cuda_device)
    if shared:
        k, kd = k.expand(B, H, Lk, D), kd.expand(B, H, Lk, D)
    ref, ref_lse = dense_attn_ref(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2))
    out, lse = full_attention_with_lse(q.to(cuda_device), kd, v.to(cuda_device), perm=perm.to(cuda_device))
    mx, mr = error_metrics(out.float().cpu().transpose(1, 2), ref)
    assert mx < 2e-2 and mr < 1e-2, (mx, mr)
    assert float((lse.cpu() - ref_lse).abs().max()) < 2e-3
    out_g, lse_g = full_attention_with_lse(q.to(cuda_device), kd, v.to(cuda_device), perm=perm.to(cuda_device), group_order=True)
    idx = perm.view(B, H, Lq).to(cuda_device)
    assert torch.equal(out_g, out.gather(2, idx.unsqueeze(-1).expand_as(out))) and torch.equal(lse_g, lse.gather(2, idx))


def _two_stream(heads, Lq, D):
    """The dispatch's choice: waves of pairs of 128-row groups, at their price, against waves of single groups."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-heads * -(-Lq // 256) // sms) * (1.5 if D == 64 else 1.7) < -(-heads * -(-Lq // 128) // sms)


def _per_head(q, k, v, **kw):
    """The same rows as launches of one head each: few groups, the gathering kernel."""
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    parts = [full_attention_with_lse(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], **kw) for h in range(q.shape[1])]
    return torch.cat([o for o, _ in parts], 1), torch.cat([l for _, l in parts], 1)


# the two-stream kernel: one key tile and several, whole and ragged, an even and an odd number of groups per head, one item per
# CTA and two
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Lq,Lk,D", [(600, 700, 128), (600, 700, 64), (513, 100, 128), (600, 128, 128), (512, 385, 64), (600, 1, 128), (4700, 300, 128), (4700, 129, 64)])
def test_dense_two_stream_kernel(cuda_device, dtype, Lq, Lk, D):
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    H = {600: 40, 513: 40, 512: 44, 4700: 13}[Lq]
    assert _two_stream(H, Lq, D) and not _two_stream(1, Lq, D)
    g = torch.Generator().manual_seed(Lq + Lk + D)
    q, k, v = (torch.randn(1, H, n, D, generator=g).to(dtype) for n in (Lq, Lk, Lk))
    qd, kd, vd = (t.to(cuda_device) for t in (q, k, v))
    out, lse = full_attention_with_lse(qd, kd, vd)
    for h in (0, H - 1):
        ref, ref_lse = dense_attn_ref(*(t[:, h:h + 1].transpose(1, 2) for t in (q, k, v)))
        mx, mr = error_metrics(out[:, h:h + 1].float().cpu().transpose(1, 2), ref)
        assert mx < 2e-2 and mr < 1e-2, (h, mx, mr)
        assert float((lse[:, h:h + 1].cpu() - ref_lse).abs().max()) < 2e-3
    o1, l1 = _per_head(qd, kd, vd)
    assert torch.equal(out, o1) and torch.equal(lse, l1)                  # the two kernels add in the same order


@pytest.mark.parametrize("dtype,D,levels", [(torch.bfloat16, 128, (0, 26, 52, 52, 78)), (torch.bfloat16, 64, (0, 26, 52, 52, 78)),
                                            (torch.float16, 128, (0, 0, 13, 13)), (torch.float16, 64, (0, 0, 13, 13))])
@pytest.mark.parametrize("H", [40, 1])
def test_dense_maximum_rises_from_tile_to_tile(cuda_device, dtype, D, levels, H):
    """Scores that rise from key tile to key tile by more than the range P has (2^24, fp16 2^12), so that the accumulator is
    rescaled while products are in flight, and values that fall by as much, so that every tile weighs the same in the output:
    a tile whose part was not rescaled, twice or too late, would dominate it.  Scores near 78 are off by 78 * 2^-20 or less
    (fp32 sums of up to 128 products): together with the rounding of P and of the output well below the tolerance."""
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    Lq, T = 600, len(levels)
    assert _two_stream(H, Lq, D) == (H > 1)
    g = torch.Generator().manual_seed(D + T)
    q, k = 0.3 * torch.randn(1, H, Lq, D, generator=g), 0.3 * torch.randn(1, H, T * 128 - 28, D, generator=g)
    v = torch.randn(1, H, T * 128 - 28, D, generator=g)
    level = torch.tensor([levels[j // 128] for j in range(k.shape[2])], dtype=torch.float32)
    q[..., 0] = 8.0
    k[..., 0] = level * (D ** 0.5 * 0.6931471805599453 / 8.0)             # 2^level in the softmax
    v *= torch.exp2((12.0 if dtype == torch.float16 else 0.0) - level).view(1, 1, -1, 1)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    qd, kd, vd = (t.to(cuda_device) for t in (q, k, v))
    out, lse = full_attention_with_lse(qd, kd, vd)
    for h in {0, H - 1}:
        ref, ref_lse = dense_attn_ref(*(t[:, h:h + 1].transpose(1, 2) for t in (q, k, v)), dtype=torch.float64)
        mx, mr = error_metrics(out[:, h:h + 1].double().cpu().transpose(1, 2), ref)
        assert mx < 3e-2 * float(ref.abs().max()) and mr < 1e-2, (h, mx / float(ref.abs().max()), mr)
        assert float((lse[:, h:h + 1].cpu() - ref_lse).abs().max()) < 2e-3
    o1, l1 = _per_head(qd, kd, vd)
    assert torch.equal(out, o1) and torch.equal(lse, l1)
    for _ in range(3):
        o2, l2 = full_attention_with_lse(qd, kd, vd)
        assert torch.equal(out, o2) and torch.equal(lse, l2)


def test_dense_inputs_with_strided_rows(cuda_device):
    """q, k, v whose last dimension is not the contiguous one: copied for the kernel, and the output is what the kernel wrote."""
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention
    g = torch.Generator().manual_seed(9)
    q, k, v = (torch.randn(1, 2, 64, n, generator=g).to(torch.bfloat16).to(cuda_device).transpose(2, 3) for n in (200, 300, 300))
    assert q.stride(-1) != 1
    assert torch.equal(full_attention(q, k, v), full_attention(q.contiguous(), k.contiguous(), v.contiguous()))

"""GPU parity: dense attention with LSE (the attention kernel's dense mode) against the fp32 oracle.

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


# edges of the two-stream kernel: one row, one key, stream B empty / one row, several items per CTA; and layouts that no
# tensor map describes (keys shared by all heads: stride 0), which take the gathering kernel
@pytest.mark.parametrize("Lq,Lk,D,shared", [(1, 1, 128, False), (128, 129, 64, False), (129, 127, 128, False), (256, 640, 64, False),
                                            (513, 300, 128, False), (5000, 200, 64, False), (300, 260, 128, True), (257, 130, 64, True),
                                            (5000, 129, 128, False), (1025, 260, 128, False), (1153, 1, 64, False)])
def test_dense_edges(cuda_device, Lq, Lk, D, shared):
    from mcsparse_b200.kernels.flash_mcsa.ops.full_attn import full_attention_with_lse
    # (more groups of 128 rows than SMs: the dense kernel; fewer: the gathering one)
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

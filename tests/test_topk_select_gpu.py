"""GPU parity: top-k selection kernel vs the CPU oracle — bit-exact on identical fp32 scores."""

import pytest
import torch

from oracle.select import select_topk_ref

pytestmark = pytest.mark.gpu


def _run(dev, scores, k_total, sink_ranges):
    from mcsparse_b200.kernels.flash_mcsa.token_sparse import select_topk_with_sinks
    return select_topk_with_sinks(scores.to(dev), k_total, sink_ranges).cpu()


@pytest.mark.parametrize("L,k_total", [(1000, 128), (4096, 512), (32760, 2048), (70000, 4096)])
def test_random_scores_exact(cuda_device, L, k_total):
    g = torch.Generator().manual_seed(L)
    scores = torch.rand(3, 2, L, generator=g) ** 8          # mass-like: many tiny values
    out = _run(cuda_device, scores, k_total, [(0, 4)])
    ref = select_topk_ref(scores, k_total, sinks=range(4))
    assert torch.equal(out, ref)


def test_ties_go_to_lowest_index(cuda_device):
    L = 5000
    g = torch.Generator().manual_seed(1)
    scores = torch.randint(0, 6, (4, L), generator=g).float() / 8        # only 6 distinct values
    scores[1] = 0.0                                                      # fully tied row
    scores[2, ::2] = -0.0                                                # -0 and +0 tie
    out = _run(cuda_device, scores, 640, [(0, 4), (100, 103)])
    ref = select_topk_ref(scores, 640, sinks=[0, 1, 2, 3, 100, 101, 102])
    assert torch.equal(out, ref)


def test_negative_and_no_sinks_and_full_row(cuda_device):
    g = torch.Generator().manual_seed(2)
    scores = torch.randn(5, 777, generator=g)
    assert torch.equal(_run(cuda_device, scores, 256, None), select_topk_ref(scores, 256))
    assert torch.equal(_run(cuda_device, scores, 777, [(0, 4)]), select_topk_ref(scores, 777, range(4)))
    assert torch.equal(_run(cuda_device, scores, 4, [(0, 4)]), select_topk_ref(scores, 4, range(4)))


def test_reference_shaped_wrapper(cuda_device):
    from mcsparse_b200.kernels.flash_mcsa.token_sparse import _select_topk_tokens
    g = torch.Generator().manual_seed(3)
    tp = torch.rand(1, 2, 3, 1024, generator=g)
    gi, gl = _select_topk_tokens(tp.to(cuda_device), 0.125, sink_ranges=[(0, 4)])
    assert tuple(gi.shape) == (1, 2, 3, 128) and gl is not None and int(gl.min()) == 1 == int(gl.max())
    assert torch.equal(gi.cpu(), select_topk_ref(tp, 128, range(4)))
    gi2, gl2 = _select_topk_tokens(tp.to(cuda_device), 0.25)
    assert tuple(gi2.shape) == (1, 2, 3, 256) and gl2 is None
    assert torch.equal(gi2.cpu(), select_topk_ref(tp, 256))


@pytest.mark.parametrize("L", [32768, 32761, 8193, 4100])
def test_rows_that_mislead_the_sample(cuda_device, L):
    """Rows that defeat the sampled lower bound of the streaming kernel (it must only cost time): one key in L / 4096 is sampled in
    rows of more than 8,192.  Winners at the sampled positions alone (the bound is too high: fewer candidates than wanted) and
    everywhere but there (too low: more than fit); ramps, NaN-heavy and constant rows, a few NaNs."""
    g = torch.Generator().manual_seed(L)
    k_total = 2048 if L > 5000 else 512
    rows = []
    rows.append(torch.arange(L).float())                                   # winners at the end
    rows.append(torch.arange(L, 0, -1).float())                            # winners at the start
    sampled = torch.zeros(L, dtype=torch.bool)
    sampled[torch.arange(4096) * L // 4096] = True
    rows.append(torch.rand(L, generator=g) * 0.5 + sampled)                # too few above the bound
    rows.append(torch.rand(L, generator=g) * 0.5 + ~sampled)               # (L > 8,192) everything not sampled above the bound
    hidden = torch.zeros(L)                                                # no winner sampled: the bound is the zeros' tie group
    pos = (~sampled if L > 8192 else sampled | ~sampled).nonzero().flatten()[: k_total + 100]
    hidden[pos] = 1.0 + torch.rand(pos.numel(), generator=g)
    rows.append(hidden)
    nan_row = torch.rand(L, generator=g)
    nan_row[torch.randperm(L, generator=g)[: L - 500]] = float("nan")      # NaN ranks highest (torch.topk): a huge tie at the top
    rows.append(nan_row)
    rows.append(torch.full((L,), 0.25))                                    # constant row
    rows.append(torch.rand(L, generator=g) ** 16)                          # mass-like
    few = torch.rand(L, generator=g)
    few[torch.randperm(L, generator=g)[:37]] = float("nan")
    rows.append(few)
    scores = torch.stack(rows)
    out = _run(cuda_device, scores, k_total, [(0, 4)])
    ref = select_topk_ref(scores, k_total, sinks=range(4))
    assert torch.equal(out, ref)


# rows around the streaming kernel's edges: every key a candidate / sampled bound (8,192), unaligned row starts (odd
# lengths), 16-bit word prefixes (131,072), budgets at which another kernel takes over
@pytest.mark.parametrize("L,k_total", [(130, 128), (8192, 2048), (8193, 2048), (16381, 9000), (33001, 128), (40000, 20000),
                                       (98279, 4096), (131072, 8192), (131073, 512)])
def test_streaming_edges(cuda_device, L, k_total):
    g = torch.Generator().manual_seed(L)
    k_total = min(k_total, L)
    rows = [torch.rand(L, generator=g) ** 12, torch.randn(L, generator=g)]
    under = torch.rand(L, generator=g)                                     # fewer than k masses survive, the rest tie at zero
    under[torch.randperm(L, generator=g)[: L - k_total // 2]] = 0.0
    rows.append(under)
    rows.append(torch.arange(L).float().flip(0))                           # winners in front
    spike = torch.full((L,), -float("inf"))                                # fewer than k finite keys
    spike[::7] = torch.rand(spike[::7].numel(), generator=g)
    rows.append(spike)
    nan_row = torch.rand(L, generator=g)
    nan_row[torch.randperm(L, generator=g)[: L // 2]] = float("nan")
    rows.append(nan_row)
    rows.append(torch.randint(0, 40, (L,), generator=g).float())           # a tie group around rank k
    scores = torch.stack(rows)
    sinks = [0, 1, 2, 3, L - 1]
    ranges = [(0, 4), (L - 1, L)]
    ref = select_topk_ref(scores, k_total, sinks=sinks)
    assert torch.equal(_run(cuda_device, scores, k_total, ranges), ref)
    shifted = torch.empty(scores.numel() + 1, device=cuda_device)[1:].view(scores.shape)   # 4-byte aligned base
    shifted.copy_(scores)
    assert torch.equal(_run(cuda_device, shifted, k_total, ranges), ref)


def test_threads_with_different_row_lengths(cuda_device):
    """Launches of one kernel with different shared-memory sizes from several threads at once."""
    import threading
    from mcsparse_b200.kernels.flash_mcsa.token_sparse import select_topk_with_sinks
    shapes = [(4100, 512), (98280, 4096), (32760, 2048), (32760, 12000), (49000, 40000), (8200, 100)]
    data = []
    for L, k in shapes:
        s = torch.rand(40, L, generator=torch.Generator().manual_seed(L + k)) ** 8
        data.append((s.to(cuda_device), k, select_topk_ref(s, k, sinks=range(4))))
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            with torch.cuda.device(cuda_device), torch.cuda.stream(torch.cuda.Stream()):
                for n in range(30):
                    s, k, ref = data[(i + n) % len(data)]
                    out = select_topk_with_sinks(s, k, [(0, 4)])
                    if n >= 24 and not torch.equal(out.cpu(), ref):
                        errors.append((i, n))
        except Exception as e:                               # noqa: BLE001 (reported below)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors


@pytest.mark.parametrize("L,k_total", [(300, 128), (9000, 1024), (32760, 28000)])          # streaming kernel (two forms), general kernel
def test_repeated_sinks_leave_no_foreign_entries(cuda_device, L, k_total):
    """The device-list entry point cannot check its sinks on the host.  Repeated ones are outside its contract; the row then holds
    fewer indices, ascending, and zeros behind them - nothing that was not written."""
    from mcsparse_b200 import _lib
    scores = torch.rand(5, L, generator=torch.Generator().manual_seed(L)) ** 8
    sinks = torch.tensor([3, 7, 7, 7], dtype=torch.int32, device=cuda_device)
    out = torch.full((5, k_total), 0x3F800000, dtype=torch.int32, device=cuda_device)
    d = scores.to(cuda_device)
    assert _lib.lib().mcs_topk_select(d.data_ptr(), out.data_ptr(), sinks.data_ptr(), 4, 5, L, k_total, torch.cuda.current_stream().cuda_stream) == 0
    out = out.cpu()
    want = select_topk_ref(scores, k_total - 2, sinks=[3, 7])
    assert torch.equal(out[:, :k_total - 2], want) and bool((out[:, k_total - 2:] == 0).all())

"""Kept start vectors of the query grouping and captured graphs: a graph must not hold the address of a tensor that the pool may
drop, so the default vectors are refused under capture, whether the pool is warm or not."""

import pytest
import torch

from mcsparse_b200.kernels.flash_mcsa import pca_group as P


class _Kept:
    """Stands in for a device tensor of the pool (no GPU needed)."""

    recorded = 0

    def numel(self):
        return 64

    def record_stream(self, stream):
        self.recorded += 1


@pytest.fixture
def capture_state(monkeypatch):
    import contextlib
    state = {"capturing": False, "asked": []}

    @contextlib.contextmanager
    def on(device):
        state["asked"].append(device)
        yield

    monkeypatch.setattr(torch.cuda, "device", on)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: None)
    return state


def test_default_start_vectors_are_refused_under_capture(capture_state):
    dev = torch.device("cuda", 0)
    pool = P._StartVectorPool()
    kept = _Kept()
    pool._entries[(0, 2, 1500, 128, 64, 0)] = kept
    assert pool.get(2, 1500, 128, 64, 0, dev) is kept and kept.recorded == 1
    capture_state["capturing"] = True
    for shape in ((2, 1500, 128, 64, 0), (2, 1600, 128, 64, 0)):           # there already; not there
        with pytest.raises(RuntimeError, match="start_vectors"):
            pool.get(*shape, dev)
    assert kept.recorded == 1 and list(pool._entries) == [(0, 2, 1500, 128, 64, 0)]
    assert set(capture_state["asked"]) == {dev}                            # the device of x, not the current one
    capture_state["capturing"] = False
    assert pool.get(2, 1500, 128, 64, 0, dev) is kept


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 96])
def test_captured_grouping(cuda_device, D, monkeypatch):
    """Under capture: the default vectors are refused with a warm and with a cold pool; given vectors are captured, and the
    replays do not depend on the pool."""
    monkeypatch.setenv("MCSPARSE_B200_CHECK", "0")                         # (the check waits for the device, which a capture refuses)
    x = torch.randn(2, 1500, D, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(cuda_device)
    sv = P.pddp_start_vectors(2, 1500, 128, D, seed=0).to(cuda_device)
    want = P.pca_group_perm(x)                                             # the pool is warm now
    torch.cuda.synchronize()
    for warm in (True, False):
        if not warm:
            P.release_start_vectors()
        g, seen = torch.cuda.CUDAGraph(), None
        with torch.cuda.graph(g):
            try:
                P.pca_group_perm(x)
            except RuntimeError as e:
                seen = str(e)
            got = P.pca_group_perm(x, start_vectors=sv)
        assert seen is not None and "start_vectors" in seen
        for _ in range(2):
            P.pca_group_perm(x)                                            # outside: kept again
            P.release_start_vectors()
            junk = torch.full((1 << 22,), 7.0, device=cuda_device)         # what the allocator hands out next
            got.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(got, want)
            del junk
    assert torch.equal(P.pca_group_perm(x), want)

"""Sort keys of the query grouping (csrc/pddp_key.cuh, compiled for the host): a key names a row of its node whatever it holds."""

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "mcsparse_b200" / "csrc"


@pytest.fixture(scope="module")
def keys(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("key")
    (d / "k.cpp").write_text(f'''
#include "{CSRC}/pddp_key.cuh"
extern "C" unsigned long long key(unsigned p, int r) {{ return mcs::sort_key(p, r); }}
extern "C" int position(unsigned long long k, int n) {{ return mcs::key_position(k, n); }}
''')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", str(d / "k.cpp"), "-o", str(d / "k.so")], check=True)
    lib = C.CDLL(str(d / "k.so"))
    lib.key.restype, lib.key.argtypes = C.c_uint64, [C.c_uint32, C.c_int32]
    lib.position.restype, lib.position.argtypes = C.c_int32, [C.c_uint64, C.c_int32]
    return lib


@pytest.mark.parametrize("size", [1, 2, 7, 128, 2048, 98280])
def test_key_names_a_row_of_its_node(keys, size):
    for r in {0, 1, size // 2, size - 1} & set(range(size)):
        for p in (0, 1, 0x80000000, 0xFFFFFFFF):
            assert keys.position(keys.key(p, r), size) == r
    # memory that nobody wrote: an earlier level's keys, padding, any bits
    g = torch.Generator().manual_seed(size)
    stale = torch.randint(-2**63, 2**63 - 1, (500,), generator=g).tolist() + [-1, 0, 2**31, 2**32 - 1, 2**31 - 1, -2**63, size, size + 1]
    assert all(0 <= keys.position(k & (2**64 - 1), size) < size for k in stale)


def test_sort_reads_rows_through_the_bound():
    """The kernel that writes the new order has no other way from a key to a row."""
    src = (CSRC / "pddp.cu").read_text()
    writes = [line for line in src.splitlines() if "perm_out[" in line and "perm_in[" in line]
    assert writes and all("key_position(" in line for line in writes), writes


@pytest.mark.gpu
@pytest.mark.parametrize("BH,N,D", [(2, 1000, 128), (3, 5000, 64), (1, 9000, 128), (2, 3000, 96)])
@pytest.mark.parametrize("poison", [0xFF, 0x7F, 0x00])
def test_grouping_with_a_raised_status_word_is_a_permutation(cuda_device, BH, N, D, poison):
    """A status word that an earlier launch left raised makes the kernels' waits give up early where they have to wait; a
    workspace full of other data shows what was not written.  Whatever the waits did, the order is one of 0 .. N-1."""
    from mcsparse_b200 import _lib
    from mcsparse_b200.kernels.flash_mcsa.pca_group import pddp_start_vectors
    lib, dev = _lib.lib(), cuda_device
    x = torch.randn(BH, N, D, generator=torch.Generator().manual_seed(N)).to(torch.bfloat16).to(dev)
    sv = pddp_start_vectors(BH, N, 128, D, 0).to(dev)
    ws = torch.full((lib.mcs_pddp_workspace_bytes(BH, N, 128),), poison, dtype=torch.uint8, device=dev)
    status = torch.full((1,), 160, dtype=torch.int32, device=dev)
    perm = torch.full((BH, N), -1, dtype=torch.int64, device=dev)
    a = _lib.PddpArgs()
    a.x, a.start_vectors, a.perm_out, a.workspace, a.workspace_bytes = x.data_ptr(), sv.data_ptr(), perm.data_ptr(), ws.data_ptr(), ws.numel()
    a.proj_levels, a.perm_levels, a.status = None, None, status.data_ptr()
    a.x_stride_bh, a.x_stride_row = x.stride(0), x.stride(1)
    a.BH, a.N, a.D, a.C, a.pow_iters, a.dtype = BH, N, D, 128, 4, _lib.MCS_DTYPE_BF16
    assert lib.mcs_pddp_perm(C.byref(a), torch.cuda.current_stream(dev).cuda_stream) == 0
    torch.cuda.synchronize(dev)
    assert torch.equal(perm.cpu().sort(dim=1).values, torch.arange(N).expand(BH, N))

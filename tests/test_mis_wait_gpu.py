"""The bounded wait of the maximal independent set's pass.

A pass gives up when the device error word is set or when nothing moves
anywhere for two seconds.  Neither can be brought about through the C ABI, so
the kernel is compiled a second time here with its control block in the
test's hands (native/mis_wait.cu): the give-up path is entered by an error
word that is set before the launch, and the words by which the pass sees that
others progress are read after it.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from pbbsbench_b200 import _capi

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def native(cuda_device, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("mis_wait") / "mis_wait.so")
    subprocess.run(["nvcc"] + _capi.NVCC_FLAGS + ["-I" + _capi.INCLUDE, "-shared", "-o", so,
                                                  os.path.join(HERE, "native", "mis_wait.cu")], check=True)
    return ctypes.CDLL(so)


def path_graph(n):
    i = np.arange(n - 1, dtype=np.uint32)
    return O.csr_symmetric(n, i, i + 1)


def on_device(off, edg):
    import torch

    d = torch.as_tensor(off.view(np.int32), device="cuda"), torch.as_tensor(edg.view(np.int32), device="cuda")
    torch.cuda.synchronize()
    return d


def args(d, n, m, flags):
    return (ctypes.c_void_p(d[0].data_ptr()), ctypes.c_void_p(d[1].data_ptr()), ctypes.c_uint32(n), ctypes.c_uint64(m),
            ctypes.c_void_p(flags.data_ptr()))


@pytest.mark.parametrize("n", [40_000, 500_003])
def test_a_set_error_word_ends_every_wait(native, n):
    """A path in id order: nearly every warp waits for the one before it when
    it looks at the error word.  All of them leave, the pass ends, and what
    was decided until then is right."""
    import torch

    off, edg = path_graph(n)
    d = on_device(off, edg)
    flags = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert native.mis_with_error_set(*args(d, n, len(edg), flags), ctypes.c_uint32(2)) == 2
    got = flags.cpu().numpy()
    want = O.mis_serial(off, edg)
    assert (got == 0).any() and (got != 0).any()
    assert np.array_equal(got[got != 0], want[got != 0])


@pytest.mark.parametrize("n", [31, 1000, 227_329, 500_003])
@pytest.mark.parametrize("stale", [0, 0xFF])
def test_every_call_shows_its_own_progress(native, n, stale):
    """A warp's progress word tells how far it is in this call, whatever the
    words held before: a finished tile always changes it, also where a warp
    has one tile and did the same one in the call before."""
    import torch

    off, edg = path_graph(n)
    d = on_device(off, edg)
    flags = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    done = np.full(1 << 16, 7, np.uint32)
    words = ctypes.c_uint32()
    assert native.mis_progress_words(*args(d, n, len(edg), flags), ctypes.c_int(stale),
                                     done.ctypes.data_as(ctypes.c_void_p), ctypes.byref(words)) == 0
    assert np.array_equal(flags.cpu().numpy(), O.mis_serial(off, edg))
    tiles = (n + 31) // 32
    warps = min(words.value // 24, tiles) * 24  # 24 warps a block, as many blocks as there are tiles at most
    last = np.arange(warps) + (np.maximum(tiles - 1 - np.arange(warps), 0) // warps) * warps
    want = np.zeros(words.value, np.uint32)
    want[:warps] = np.where(np.arange(warps) < tiles, last + 1, 0)
    assert np.array_equal(done[: words.value], want)

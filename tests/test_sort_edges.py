"""Radix sorts against the oracle's stable sort: at the edges of the sort that
one cluster of blocks does in one launch (of a block, of the keys a thread holds,
of the cluster) and of the tiled sort's two tiles, with short keys, few distinct
keys and under stream capture."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sort(L, keys, bits, capture=False):
    import torch

    n = len(keys)
    dk = torch.from_numpy(keys.view(np.int32)).to("cuda")
    do = torch.full((n + 32,), -1, dtype=torch.int32, device="cuda")
    need = C.c_size_t()
    assert L.vsim_radix_sort_u32(dk.data_ptr(), do.data_ptr(), n, bits, None, C.byref(need), None) == 0
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")

    def run():
        st = torch.cuda.current_stream().cuda_stream
        assert L.vsim_radix_sort_u32(dk.data_ptr(), do.data_ptr(), n, bits, temp.data_ptr(), C.byref(need), st) == 0

    if capture:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        for _ in range(2):
            do.fill_(-1)
            graph.replay()
    else:
        run()
    torch.cuda.synchronize()
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys)  # input untouched
    out = do.cpu().numpy()
    assert (out[n:] == -1).all()
    return out[:n].view(np.uint32)


# A block holds 512 keys for each key a thread, a cluster 16 blocks of at most 6
# keys a thread (49,152); then tiles of 4096 keys, and past two tiles an SM
# (304 on 152 of them) of 6144.
SIZES = [1, 31, 33, 511, 512, 513, 8191, 8192, 8193, 16384, 16385, 30011, 32768, 32769, 49151, 49152, 49153, 53248,
         65537, 120001, 304 * 4096, 304 * 4096 + 1, 203 * 6144, 203 * 6144 + 1, 1_300_001]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits", [32, 8, 9, 1])
def test_sort_matches_stable_sort(vsimlib, gpu, n, bits):
    import pyoracle

    rng = np.random.default_rng(n * 40 + bits)
    keys = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32)
    assert np.array_equal(sort(vsimlib.lib(), keys, bits), pyoracle.stable_sort(keys, bits))


@pytest.mark.parametrize("n", [1025, 30011, 49152, 131072])
@pytest.mark.parametrize("kind", ["equal", "few", "sorted", "reversed"])
def test_sort_of_skewed_keys(vsimlib, gpu, n, kind):
    import pyoracle

    rng = np.random.default_rng(n)
    keys = {"equal": np.full(n, 0xFFFFFFFF, np.uint32),
            "few": rng.choice(np.array([0, 255, 256, 0x80000000], np.uint32), n),
            "sorted": np.arange(n, dtype=np.uint32) * 3,
            "reversed": np.arange(n, dtype=np.uint32)[::-1].copy()}[kind]
    assert np.array_equal(sort(vsimlib.lib(), keys, 32), pyoracle.stable_sort(keys, 32))


def test_sort_under_capture(vsimlib, gpu):
    import pyoracle

    keys = np.random.default_rng(5).integers(0, 2 ** 32, 30011, dtype=np.uint64).astype(np.uint32)
    assert np.array_equal(sort(vsimlib.lib(), keys, 32, capture=True), pyoracle.stable_sort(keys, 32))

"""The argsort at the edges of its scatter tiles (4096 keys; 512-thread blocks up to 296 tiles, 256-thread
blocks beyond), against a stable argsort: sizes around a tile, around the change of block, a count below
the capacity, keys of all ones (which pad a last tile) and keys of one digit."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk


def argsort(keys, bits, capacity=None):
    import torch

    n = len(keys)
    capacity = n if capacity is None else capacity
    padded = np.full(capacity, 3, np.uint32)
    padded[:n] = keys
    d = torch.from_numpy(padded.view(np.int32)).cuda()
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    order = torch.full((capacity,), -1, dtype=torch.int32, device="cuda")
    work = torch.empty((sk.sort_workspace_bytes(capacity),), dtype=torch.uint8, device="cuda")
    error = torch.zeros((1,), dtype=torch.int32, device="cuda")
    sk.radix_argsort_device(d.data_ptr(), count.data_ptr(), capacity, bits, order.data_ptr(), work.data_ptr(),
                            work.numel(), error.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(error.item()) == 0
    got = order.cpu().numpy()
    assert np.all(got[n:] == -1)  # nothing is written past the count
    return got[:n]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 8193, 296 * 4096, 296 * 4096 + 1, 300 * 4096 - 7])
@pytest.mark.parametrize("bits", [16, 32])
def test_sizes_around_the_tiles(cuda_device, n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[rng.random(n) < 0.1] = (1 << bits) - 1  # every digit 255
    assert np.array_equal(argsort(keys, bits), np.argsort(keys, kind="stable"))


@pytest.mark.gpu
@pytest.mark.parametrize("n,capacity", [(5_000, 20_000), (100, 1_300_000), (0, 9_000)])
def test_a_count_below_the_capacity(cuda_device, n, capacity):
    keys = np.random.default_rng(5).integers(0, 1 << 16, n, dtype=np.uint32)
    assert np.array_equal(argsort(keys, 16, capacity), np.argsort(keys, kind="stable"))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [0, 0x41A00000, 0xFFFFFFFF])
def test_keys_that_are_all_equal_keep_their_order(cuda_device, value):
    keys = np.full(70_001, value, np.uint32)
    assert np.array_equal(argsort(keys, 32), np.arange(70_001))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 2049, 8192, 8193, 16_385, 20_011, 32_767, 32_768, 32_769])
@pytest.mark.parametrize("bits", [16, 32])
def test_sizes_around_the_one_launch_sort(cuda_device, n, bits):
    """One cluster of 1, 2, 4 or 8 blocks of 1 to 4 rows (cluster_sort.cu) up to 32,768 keys."""
    rng = np.random.default_rng(n * 3 + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[rng.random(n) < 0.2] = keys[0]
    assert np.array_equal(argsort(keys, bits), np.argsort(keys, kind="stable"))
    assert np.array_equal(argsort(keys[: n // 2], bits, n), np.argsort(keys[: n // 2], kind="stable"))

"""The pair sort at the edges of its passes: full and partial tiles, warps whose keys share a digit beside
warps whose keys do not, unaligned inputs, outputs that are the inputs, and one pass against several.
The oracle is numpy's stable sort; results are whole numbers and equal."""
from __future__ import annotations

import numpy as np
import pytest

import master_thesis_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    assert t.cuda.is_available(), "a CUDA GPU is required"
    return t


def keys_of(kind, n, bits):
    rng = np.random.default_rng(n * 31 + bits)
    space = 1 << bits
    if kind == "uniform":  # every digit shared by whole warps
        return np.full(n, space - 1, np.int64)
    if kind == "runs":  # consecutive keys with jumps: low digits differ, high ones are shared or split a warp
        start = rng.integers(0, space, 1 + n // 97)
        i = np.arange(n)
        return (start[i // 97] + i % 97) % space
    return rng.integers(0, space, n)


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 12289, 70001])
@pytest.mark.parametrize("bits,rb", [(7, 8), (8, 8), (17, 8), (20, 9), (19, 10), (32, 11)])
@pytest.mark.parametrize("kind", ["uniform", "runs", "random"])
@pytest.mark.parametrize("place", ["apart", "in_place", "unaligned"])
def test_sort_pairs_forms(torch, place, kind, bits, rb, n):
    k = keys_of(kind, n, bits).astype(np.uint32)
    v = np.arange(n, dtype=np.uint32)[::-1].copy()
    order = np.argsort(k, kind="stable")
    off = 1 if place == "unaligned" else 0
    kin = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    vin = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    kin[off:off + n] = torch.from_numpy(k.view(np.int32)).cuda()
    vin[off:off + n] = torch.from_numpy(v.view(np.int32)).cuda()
    ki, vi = kin[off:off + n], vin[off:off + n]
    ko, vo = (ki, vi) if place == "in_place" else (torch.zeros_like(ki), torch.zeros_like(vi))
    nb = T.lib().tecto_sort_scratch_bytes_radix(n, bits, rb)
    scr = torch.empty(nb, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    T.check(T.lib().tecto_sort_pairs_radix(ki.data_ptr(), vi.data_ptr(), ko.data_ptr(), vo.data_ptr(), n, bits, rb,
                                           scr.data_ptr(), nb, None), "tecto_sort_pairs_radix")
    np.testing.assert_array_equal(ko.cpu().numpy().view(np.uint32), k[order])
    np.testing.assert_array_equal(vo.cpu().numpy().view(np.uint32), v[order])

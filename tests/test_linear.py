"""Which kernel a projection goes to: by its weight alone.  On the CPU."""
import pytest
import torch

from spyinfer_b200 import kernels
from spyinfer_b200.parts.linear import Linear


@pytest.mark.parametrize("N,K,split", [(256, 8, False), (256, 56, False), (256, 64, True), (33, 64, True), (32, 64, False), (256, 100, False), (256, 104, True)])
def test_products_of_the_float32_path(N, K, split, monkeypatch):
    """Weights of short rows (fewer than 64 terms), few rows or rows that are no multiple of 16 bytes stay with the CUDA-core product, and so do such
    parts of a weight that does not."""
    went = []
    monkeypatch.setattr(kernels, "gemm_split", lambda x, w, out: went.append(("split", tuple(w.shape))) or out)
    monkeypatch.setattr(kernels, "gemm_simt", lambda x, w, out: went.append(("simt", tuple(w.shape))) or out)
    linear = Linear(torch.zeros(N, K, dtype=torch.bfloat16), torch.float32)
    for rows in (1, 300):
        linear(torch.zeros(rows, K))
    assert went == [("split" if split else "simt", (N, K))] * 2 and ("gemm_split" in linear.modules()) == split
    whole = Linear(torch.zeros(300, 256, dtype=torch.bfloat16), torch.float32)
    for rows, cols in (((0, N), (0, K)), ((0, N), (8, 8 + K))):
        went.clear()
        whole.part(torch.zeros(2, K), rows=rows, cols=cols)
        assert went == [("split" if split else "simt", (N, K))]


def test_a_weight_of_more_rows_than_the_split_products_grid_takes():
    """Such a weight (made without memory) stays with the CUDA-core product, which takes any number of rows."""
    for rows, split in ((65535 * 64, True), (65535 * 64 + 1, False)):
        assert Linear(torch.empty(rows, 64, dtype=torch.bfloat16, device="meta"), torch.float32).split == split

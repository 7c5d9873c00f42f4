"""The rules that choose a kernel by sizes, at sizes on both sides of their lines (host logic, no GPU)."""

from __future__ import annotations

import pytest

from mini_gpt_inference_b200.kernels.ops import CudaOps


@pytest.mark.parametrize("m,n,k,cluster", [
    (17, 2304, 768, True), (32, 3072, 768, True), (32, 6400, 1600, True), (17, 8192, 2048, True), (32, 50304, 512, False),
    (33, 2304, 768, False), (64, 128, 4096, True), (64, 512, 2048, True), (64, 512, 512, False), (64, 1024, 2048, True),
    (64, 1024, 1024, False), (33, 1600, 6400, False)])
def test_projections_of_17_to_64_tokens(m, n, k, cluster):
    """Up to 32 tokens every matrix but the head's goes to the kernel that cuts K over a cluster, beyond only short and long ones."""
    assert CudaOps._cluster_pays(m, n, k) is cluster

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


@pytest.mark.parametrize("entries,experts,width,inner,few", [
    (128, 32, 512, 128, True), (64, 64, 512, 128, True), (128, 64, 512, 128, False), (128, 64, 1024, 256, False),
    (128, 64, 2048, 512, True), (2, 128, 512, 128, False), (128, 128, 1024, 1024, True), (2, 256, 1024, 1024, False)])
def test_experts_of_few_tokens(entries, experts, width, inner, few):
    """A CTA of every expert is started: not with many experts of little work."""
    assert CudaOps._moe_few_pays(entries, experts, width, inner) is few


@pytest.mark.parametrize("entries,experts,width,inner,tensor_cores", [
    (6144, 9, 1024, 1024, True), (64 * 9 - 1, 9, 1024, 1024, False), (800, 9, 1024, 1024, True), (512, 4, 1024, 1024, False),
    (768, 4, 1024, 1024, True), (32 * 32, 32, 1024, 2048, False), (64 * 32, 32, 1024, 2048, True), (4096, 16, 1024, 512, False),
    (130, 8, 512, 256, False), (4096, 64, 512, 256, False)])
def test_experts_of_many_tokens(entries, experts, width, inner, tensor_cores):
    """Tiles of 128 rows: where an expert has 64 rows and more, of large matrices, and there is work for all SMs."""
    assert CudaOps._moe_tc_pays(entries, experts, width, inner) is tensor_cores

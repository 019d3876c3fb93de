"""Scratch of the plain replay where it just fits the 32 MiB of the allocation-free entry."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_exactly_32_mib(bw, torch_cuda):
    """Two sweep CTAs' blocks over 149 keys and 284,710 states: exactly 32 MiB with the
    coarse blocks and the plain tour that the entry took when its size was set."""
    parent = torch_cuda.zeros(284_710, dtype=torch_cuda.int32, device="cuda")
    assert bw.Replay(parent, 149, 16_422_564, 9_083_838).workspace.numel() <= 32 << 20

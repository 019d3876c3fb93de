"""Scratch of the plain replay: where it just fits the 32 MiB of the allocation-free entry,
and over wide key domains with few events."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_exactly_32_mib(bw, torch_cuda):
    """Two sweep CTAs' blocks over 149 keys and 284,710 states: exactly 32 MiB with the
    coarse blocks and the plain tour that the entry took when its size was set."""
    parent = torch_cuda.zeros(284_710, dtype=torch_cuda.int32, device="cuda")
    assert bw.Replay(parent, 149, 16_422_564, 9_083_838).workspace.numel() <= 32 << 20


@pytest.mark.parametrize("S,C,E,Q,mib", [(300, 262_144, 1000, 1_000_000, 160),
                                         (300_000, 262_144, 1000, 5000, 300),
                                         (284, 2_261_068, 41, 114_912, 180)])
def test_rows_of_wide_domains(bw, torch_cuda, S, C, E, Q, mib):
    """Blocks are not cut so fine that their dense rows outweigh their work (266, 401 and 248
    MiB with as many blocks as the work alone allows)."""
    parent = torch_cuda.zeros(S, dtype=torch_cuda.int32, device="cuda")
    assert bw.Replay(parent, C, E, Q, path="general").workspace.numel() < mib << 20

"""CPU enumeration of shared-memory reads beside those of test_bank_layout.py: the energies' half-pair buffers in the
contraction launch (ozaki.cu, fused_energies), the exchange tiles of diagonal pairs (fused_tma.cu, xch_off), and the k4
step of a contraction's last chunk (fused_tma.cu, quarter_products), which does have conflicts.  A warp's 64-bit
accesses are served per half-warp: free of conflicts when its lanes touch distinct 8-byte slots of the 128-byte line, or
the same address."""
from collections import defaultdict

import pytest

PERM = [0, 6, 1, 7, 2, 4, 3, 5]


def _ways(addresses):
    """Wavefronts that one half-warp's addresses take."""
    slots = defaultdict(set)
    for a in addresses:
        slots[(a // 8) % 16].add(a)
    return max(len(v) for v in slots.values())


@pytest.mark.parametrize("half_warp", range(8))  # 128 energy threads
def test_energy_half_buffers_are_read_without_conflicts(half_warp):
    first, second, row, entry = [], [], [], []
    for te in range(16 * half_warp, 16 * half_warp + 16):
        r = te & 15
        c = (te >> 4) ^ (r >> 3)
        first.append(c * 128 + (((r >> 1) ^ c) << 4) + ((r & 1) << 3))
        second.append(r * 64 + (((c >> 1) ^ ((r >> 1) & 3)) << 4) + ((c & 1) << 3))
        row.append(8 * r)
        entry.append(8 * c)
    assert _ways(first) == 1 and _ways(second) == 1 and _ways(row) == 1 and _ways(entry) == 1
    assert len(set(first)) == 16 and len(set(second)) == 16


def _xch(row, col):
    return 8 * (row * 32 + (col ^ ((row & 3) << 2)))


@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("e", range(4))
def test_exchange_tiles_are_written_and_read_without_conflicts(half, e):
    writes, reads = [], []
    for lane in range(16 * half, 16 * half + 16):
        g, t = lane >> 2, lane & 3
        row, col = PERM[g] + (8 if e & 2 else 0), PERM[2 * t + (e & 1)]
        writes.append(_xch(row, col))
        reads.append(_xch(col, row))
    assert _ways(writes) == 1 and _ways(reads) == 1


@pytest.mark.parametrize("half", [0, 1])
def test_the_k4_step_reads_both_panel_kinds_in_two_wavefronts(half):
    kmajor, xmajor = [], []
    for lane in range(16 * half, 16 * half + 16):
        x, t = PERM[lane >> 2], lane & 3
        kmajor.append(t * 128 + (((x >> 1) ^ t) << 4) + ((x & 1) << 3))
        xmajor.append(x * 128 + (((t >> 1) ^ x) << 4) + ((t & 1) << 3))
    assert _ways(kmajor) == 2 and _ways(xmajor) == 2

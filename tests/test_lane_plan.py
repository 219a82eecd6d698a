"""How the feature-per-bank histogram pass cuts a table into document chunks, from sizes alone (no GPU)."""
import ctypes

import numpy as np
import pytest

SMS, SMEM = 148, 227 * 1024 - 64           # SMs and dynamic shared memory of a block


def _plan(n, F, bins, share, level):
    """[(document chunks, feature groups)] of the bundles of a level."""
    from catboost_b200.ops import native
    G = (F + 3) // 4
    gb = np.full(G, (bins + 3) // 4 * 4, dtype=np.int32)
    sh = np.full(G, share, dtype=np.float32)
    chunks, groups = np.zeros(G, dtype=np.int32), np.zeros(G, dtype=np.int32)
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    k = native.cuda_lib().cb_lane_plan_query(n, G, P(gb), P(sh), level, SMS, SMEM, G, P(chunks), P(groups))
    return list(zip(chunks[:k].tolist(), groups[:k].tolist()))


@pytest.mark.parametrize("n,F", [(1, 9), (10_500_000, 28), (100_000_000, 100), (20_000_000, 2000), (50_000_000, 1000), ((1 << 28) - 1, 12)])
@pytest.mark.parametrize("bins,share", [(129, 1.0 / 129), (129, 0.5), (256, 0.3), (2, 0.5), (32, 0.4)])
def test_no_cell_receives_so_many_documents_that_small_values_round_away(n, F, bins, share):
    """The scale is 2^31 / (documents of the fullest cell): at least 2^14 steps whatever the shape, 2^16 at level 0."""
    for level in range(9):
        plan = _plan(n, F, bins, share, level)
        assert sum(g for _, g in plan) == (F + 3) // 4
        blocks = (n + 1663) // 1664
        for chunks, _ in plan:
            assert 1 <= chunks <= min(max(blocks, 1), 4096)
            fullest = max(share, 1.0 / 32.0) * n / chunks
            if chunks < min(blocks, 4096):
                assert fullest <= (1 << (15 if level == 0 else 17)), (level, chunks, fullest)


def _bytes(n, F, bins, depth, share=1.0 / 64):
    from catboost_b200.ops import native
    G = (F + 3) // 4
    gb = np.full(G, (bins + 3) // 4 * 4, dtype=np.int32)
    sh = np.full(G, share, dtype=np.float32)
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    return native.cuda_lib().cb_lane_bytes(n, G, P(gb), P(sh), depth, SMS, SMEM)


@pytest.mark.parametrize("n,F", [(10_500_000, 28), (50_000_000, 1000), (20_000_000, 2000), (100_000_000, 800)])
def test_device_memory_is_the_second_copy_and_little_else(n, F):
    """Scratch is for the work items in flight: it must not grow with rows x row blocks (12 bytes each would be 19 GB at 50M x 1000)."""
    copy = n * ((F + 3) // 4) * 4
    assert copy <= _bytes(n, F, 129, 6) <= 1.15 * copy + (1 << 30)


@pytest.mark.parametrize("n,F", [(10_500_000, 4), (10_500_000, 8), (1 << 28, 28)])
def test_no_memory_for_a_pass_that_no_level_takes(n, F):
    assert _bytes(n, F, 129, 6) == 0


@pytest.mark.parametrize("n,F,bins,level", [(1_200_000, 28, 256, 9), (1_200_000, 100, 256, 7), (4_000_000, 100, 256, 7)])
def test_slot_passes_that_come_in_whole_multiples_leave_few_sms_idle(n, F, bins, level):
    """86 passes of one bundle as 86 items would leave 62 of 148 SMs without work."""
    items = 0
    for chunks, groups in _plan(n, F, bins, 1.0 / bins, level):
        lanes = 64 if groups > 4 else 32
        slots = min((SMEM // 4 - 26 * 256) // (bins * lanes + 64), 1 << (level - 1))
        items += chunks * -(-(1 << (level - 1)) // slots)
    assert items / (-(-items // SMS) * SMS) >= 0.85, items

"""What the scans over chunks of sixteen tokens refuse before they launch anything: their entry point is called without a device."""
from __future__ import annotations

import ctypes

import pytest

GATED_DELTA, DELTA_RULE, CHANNEL_DECAY, HEAD_DECAY = range(4)
SHAPE = -2


def _call(mode, H, G, D, Dv, stride, cols, gate_stride):
    """No pointer is looked at before the sizes are: 16 rows of one segment, and no device behind them."""
    from kvcache_b200.kernels.api import _Library
    p = ctypes.c_void_p(1 << 20)
    return _Library("scan_chunk").kvb_chunk_scan(mode, p, stride, *cols, G, p, gate_stride, 1.0, p, p, p, p, p, 16, 1, H, D, Dv, 2, p, p, None)


@pytest.mark.parametrize("mode,H,G,D,Dv,stride,cols,gate_stride", [
    (GATED_DELTA, 6, 4, 64, 64, 2 * 4 * 64 + 6 * 64, (0, 256, 512), 6 * 64 + 6),        # heads that do not share evenly
    (HEAD_DECAY, 6, 4, 64, 64, 6 * 64 + 2 * 4 * 64, (6 * 64 + 256, 6 * 64, 0), 12),
    (GATED_DELTA, 2, 4, 64, 64, 2 * 4 * 64 + 2 * 64, (0, 256, 512), 2 * 64 + 2),        # more groups than heads
    (GATED_DELTA, 2, 0, 64, 64, 128, (0, 0, 0), 130),
    (CHANNEL_DECAY, 2, 2, 64, 128, 512, (0, 128, 256), 127),                            # decays that are no rows of their own
    (CHANNEL_DECAY, 2, 2, 64, 128, 512, (0, 128, 256), 129),
    (GATED_DELTA, 2, 2, 64, 64, 384, (0, 128, 256), 2 * 64 + 1),                        # gates that end too early
    (DELTA_RULE, 2, 2, 64, 64, 384, (0, 128, 256), 3 * 128 - 1),
    (HEAD_DECAY, 2, 2, 64, 64, 384, (256, 128, 0), 3),
    (GATED_DELTA, 2, 2, 64, 64, 383, (0, 128, 256), 2 * 64 + 2),                        # columns beyond the row
    (DELTA_RULE, 2, 2, 64, 64, 384, (0, 257, 256), 3 * 128),
    (DELTA_RULE, 2, 2, 64, 64, 384, (-1, 128, 256), 3 * 128),
])
def test_sizes_that_do_not_fit_are_refused(mode, H, G, D, Dv, stride, cols, gate_stride):
    assert _call(mode, H, G, D, Dv, stride, cols, gate_stride) == SHAPE

"""Gates of chunked matrix memories over portions of about one and two rounds of 1,024 tokens: against the plain recurrence in
float64, and cut into shorter portions."""

import pytest
import torch

from test_dedizen_kernels_gpu import close, memory_case, run_memory

pytestmark = pytest.mark.gpu


def test_portions_around_the_rounds():
    H, d, dv, lens = 2, 32, 48, [1023, 1024, 1025, 2100]
    xs, want, extra = memory_case(H, d, dv, lens, 11, True)
    whole = run_memory(H, d, dv, xs, extra, [[n] for n in lens], True, True, torch.float32, slots=[1, 5, 0, 3])
    cut = run_memory(H, d, dv, xs, extra, [[511, 512], [1000, 24], [1024, 1], [900, 1200]], True, True, torch.float32,
                     slots=[1, 5, 0, 3], decode=False)
    for r in range(len(lens)):
        # (the chunks' tolerance: what float32 sums and pairs of bfloat16 lose)
        assert close(whole[r], want[r], 1e-3) and close(cut[r], want[r], 1e-3), lens[r]
        assert close(whole[r][-40:], want[r][-40:], 1e-3)

"""How long the bounded waits last: on a word that says a wait has run out already, and in items that are long."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa import _lib

DEV = "cuda:0"


def test_waits_of_a_launch_that_has_failed_are_short():
    L = _lib.lib()
    word = torch.zeros(4, dtype=torch.int32, device=DEV)

    def seconds():
        torch.cuda.synchronize()
        t = time.perf_counter()
        assert L.fsa_debug_wait_timeout(_lib.ptr(word), _lib.current_stream(word.device)) == 0
        torch.cuda.synchronize()
        return time.perf_counter() - t

    first, second = seconds(), seconds()      # 400e6 and 6.25e6 cycles: 0.2 s and 3 ms at 1.965 GHz
    assert int(word[0]) == 1 and first > 0.19 and second < 0.1, (first, second)

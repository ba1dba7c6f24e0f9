"""gfe_device_errors takes and clears the caller's error word: one thread, and more threads at once than the library
keeps host words (64), each with its own word and stream."""
import threading

import pytest
import torch

from iron_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_threads", [1, 64, 80])
def test_every_thread_takes_its_own_bits(gfe_cuda, n_threads):
    wrong = []
    start = threading.Barrier(n_threads)

    def work(i):
        torch.cuda.set_device(gfe_cuda)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            word = torch.zeros(1, dtype=torch.int32, device=gfe_cuda)
            _lib.set_thread_error_word(word)
            try:
                start.wait(timeout=60)
                for k in range(10):
                    word.fill_(1 + (i + k) % 15)
                    got, again = _lib.device_errors(stream), _lib.device_errors(stream)
                    if got != 1 + (i + k) % 15 or again != 0 or int(word.item()) != 0:
                        wrong.append((i, k, got, again))
            finally:
                _lib.set_thread_error_word(None)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n_threads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert _lib.device_errors() == 0

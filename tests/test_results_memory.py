"""Memory of results (Engine._logits_array): used again once nobody holds a view, of whatever kind, and never before."""
import threading
from collections import deque

import numpy as np
import torch

from leafcutterllm_b200.engine import Engine


def engine(vocab=1000):
    eng = Engine.__new__(Engine)
    eng._h, eng._memory, eng.vocab_size = None, deque(maxlen=2), vocab
    return eng


def test_memory_is_used_again_when_the_last_view_is_gone():
    eng = engine()
    first = eng._logits_array(2)
    view = first[1:, ::2]
    del first
    for hold in (lambda a: a[0][3:], np.asarray, torch.from_numpy, memoryview, lambda a: a.base, lambda a: a.reshape(-1).T):
        held = hold(eng._logits_array(2))
        for _ in range(3):
            other = eng._logits_array(2)
            assert not np.shares_memory(np.asarray(held), other) and not np.shares_memory(view, other)
        del held
    del view
    assert len({eng._logits_array(2).ctypes.data for _ in range(6)}) <= 2
    assert eng._logits_array(3).shape == (3, 1000) and eng._logits_array(2).flags.writeable


def test_results_of_several_threads_do_not_share_memory():
    eng, wrong = engine(64), []

    def work(k):
        for i in range(3000):
            a = eng._logits_array(1)
            a[:] = k * 10000 + i
            b = eng._logits_array(1)
            b[:] = -1
            if not (a == k * 10000 + i).all():
                wrong.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

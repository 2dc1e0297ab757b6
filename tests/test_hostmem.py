"""The pool of result arrays on the host: threads, forked processes."""
import gc
import os
import threading

import numpy as np

from milton_gb300 import hostmem


def test_a_forked_process_reads_and_takes_results():
    a = hostmem.empty((1 << 17,), np.float64)
    a[:] = 3.0
    held, done = threading.Event(), threading.Event()

    def hold():
        with hostmem._lock:
            held.set()
            done.wait(30)

    t = threading.Thread(target=hold)
    t.start()
    held.wait(30)
    pid = os.fork()
    if pid == 0:
        ok = bool(np.all(a == 3.0))
        b = hostmem.empty((1 << 17,), np.float64)
        b[:] = 4.0
        a[:] = 5.0
        del b
        gc.collect()
        os._exit(0 if ok and hostmem.empty((1 << 17,), np.float64).shape == (1 << 17,) else 1)
    done.set()
    t.join()
    assert os.waitpid(pid, 0)[1] == 0
    assert np.all(a == 3.0)


def test_threads_never_share_a_live_block():
    bad = []

    def work(k):
        for i in range(200):
            x = hostmem.empty((1 << 15,), np.float64)
            x[:] = k + i * 100.0
            y = x[3:9]
            del x
            if not np.all(y == k + i * 100.0):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    gc.collect()
    assert not bad and hostmem._total <= hostmem.LIMIT

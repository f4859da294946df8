"""The native half of the torch front end (csrc/host_binding.cpp) among several threads of one program."""
import sys
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_calls_let_other_threads_run(ctx):
    """With a switch interval of half a minute a thread gets the interpreter only where another gives it up: the calls of
    this loop do, so the waiting thread runs while it lasts.  (Results go to given tensors: torch gives the interpreter up
    when it frees one.)"""
    q = torch.randn((1, 1, 16, 32), device="cuda")
    o, lse = ctx.attn_fwd(q, q, q)
    torch.cuda.synchronize()
    gate, ran = threading.Lock(), []
    gate.acquire()
    t = threading.Thread(target=lambda: (gate.acquire(), ran.append(True)))
    t.start()
    time.sleep(0.1)                      # the thread waits at the gate
    interval = sys.getswitchinterval()
    sys.setswitchinterval(30)
    try:
        gate.release()
        for _ in range(5000):
            ctx.attn_fwd(q, q, q, out=o, lse=lse)
            if ran:
                break
        during = bool(ran)
    finally:
        sys.setswitchinterval(interval)
    t.join()
    assert during

"""Calls of different shapes from several host threads at once."""
import threading

import pytest
import torch

from augurv2_b200 import _native as N
from augurv2_b200 import hlrb as H

pytestmark = pytest.mark.gpu


def test_threads_with_different_shapes():
    """Kernels whose shared memory depends on the shape, launched by two
    threads with a small and a large one: every launch is accepted, and the
    results are those of the calls made alone."""
    shapes = [(8, 16), (1024, 16)]
    surs, thetas, alone = [], [], []
    for D, C in shapes:
        gen = torch.Generator("cuda").manual_seed(D)
        sur = H.MlpSurrogate(D, 64, 64, seed=D)
        theta = torch.randn(C, D, device="cuda", generator=gen)
        surs.append(sur)
        thetas.append(theta)
        alone.append(sur.predict(theta, torch.empty_like(theta)).clone())
    torch.cuda.synchronize()
    L, p = N.lib(), N.ptr
    refused, results = [], [None] * len(shapes)
    go = threading.Barrier(len(shapes))

    def call(i):
        D, C = shapes[i]
        s, theta, out = surs[i], thetas[i], torch.empty_like(thetas[i])
        st = torch.cuda.Stream()
        args = (H.C.byref(s.desc), C, p(theta), D, p(s.mu), p(s.inv_s), p(s.a), p(s.h), p(s.o), p(out), D, N.stream_ptr(st))
        go.wait()
        for _ in range(20000):
            rc = L.ab_sur_predict(*args)
            if rc != 0:
                refused.append((shapes[i], N.last_error()))
                break
        st.synchronize()
        results[i] = out

    threads = [threading.Thread(target=call, args=(i,)) for i in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not refused, refused
    for got, want in zip(results, alone):
        assert torch.equal(got, want)

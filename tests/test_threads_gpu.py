"""Calls of one kind with different sizes from several host threads: what a call
sets for its own launch must not disturb another thread's.  The threads call the
C interface (ctypes releases the interpreter lock) with everything prepared, so
that they spend their time between a kernel's set-up and its launch; before the
limit of a kernel's dynamic shared memory was the same for every call, about one
call in a thousand was refused."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cle():
    import pyclesperanto_prototype_b200 as m
    from pyclesperanto_prototype_b200 import _build
    _build.build()
    return m


# name: C function, shapes of source and destination, the scalar arguments of two
# calls that launch the same kernel with different dynamic shared memory above
# 48 KB, bytes of workspace (none: the function takes no workspace)
CALLS = {
    "blur": ("cle_gaussian_blur", (32, 24, 24), (32, 24, 24), [(0.0, 0.0, 10.0), (0.0, 0.0, 7.0)], 1 << 20),
    "box": ("cle_maximum_box", (820, 8), (820, 8), [(0.0, 400.0, 0.0), (0.0, 300.0, 0.0)], 1 << 20),
    "top_hat": ("cle_top_hat_box", (32, 12, 12), (32, 12, 12), [(2.0, 2.0, 24.0), (2.0, 2.0, 16.0)], 1 << 20),
    "histogram": ("cle_histogram", (8, 64), None, [(50000, 0.0, 1000.0, 0), (13000, 0.0, 1000.0, 0)], 1 << 22),
    "neighbours": ("cle_average_distance_of_n_distances", (101, 101), (1, 101), [(100, 1), (97, 1)], None),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_two_sizes_from_eight_threads(cle, name):
    from pyclesperanto_prototype_b200 import _lib
    lib = _lib.load()
    fn, src, dst, args, scratch = CALLS[name]
    image = torch.from_numpy(np.random.default_rng(3).uniform(0, 1000, src).astype(np.float32)).cuda()

    def prepare(k, stream):
        out = torch.zeros(dst or (args[k][0],), device="cuda")
        a, d = _lib.tensor_desc(image), _lib.tensor_desc(out)
        ws = torch.empty(scratch or 16, dtype=torch.uint8, device="cuda")
        tail = (ws.data_ptr(), ws.numel(), stream) if scratch else (stream,)
        if scratch is None:      # source, scalars, destination
            c = (_lib.ref(a),) + args[k] + (_lib.ref(d),) + tail
        else:
            c = (_lib.ref(a), _lib.ref(d)) + args[k] + tail
        return c, out, (a, d, ws)

    want = []
    for k in (0, 1):
        c, out, keep = prepare(k, torch.cuda.current_stream().cuda_stream)
        _lib.check(getattr(lib, fn)(*c), fn)
        want.append(out)
    streams = [torch.cuda.Stream() for _ in range(8)]
    ready = [prepare(i % 2, s.cuda_stream) for i, s in enumerate(streams)]
    torch.cuda.synchronize()
    refused = [0] * len(ready)

    def work(i):
        f, c = getattr(lib, fn), ready[i][0]
        for _ in range(6000):
            if f(*c):
                refused[i] += 1

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(ready))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert sum(refused) == 0
    for i, (_, out, _) in enumerate(ready):
        assert torch.equal(out, want[i % 2])

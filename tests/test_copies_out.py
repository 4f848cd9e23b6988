"""Maps copied to the host through pinned halves: every byte arrives, for sizes
around the smallest that is staged and around the halves, into memory at any
alignment, into pinned memory, and from more threads than there are kept
blocks."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(n, seed):
    from relight_b200.device import DeviceMap
    color = np.random.default_rng(seed).random((n, 3)).astype(np.float32)
    m = DeviceMap(0, n, 1)
    m.upload(color=color)
    return m, color


@pytest.mark.parametrize("n", [1, 2730, 2731, 43690, 43691, 87381, 87382, 131073, 500001])
def test_encoded_bytes(cuda, n):
    import torch
    from relight_b200 import _abi
    m, color = _map(n, n)
    raw = np.frombuffer(color.tobytes(), np.uint8)
    assert np.array_equal(m.encode(0), raw)
    assert np.array_equal(m.download(fields=("color",))["color"], color)
    buf = np.full(12 * n + 32, 7, np.uint8)
    _abi.check(_abi.lib().rl_map_encode(m.handle, 0, C.c_void_p(buf.ctypes.data + 13), None))
    assert np.array_equal(buf[13:13 + 12 * n], raw) and (buf[:13] == 7).all() and (buf[13 + 12 * n:] == 7).all()
    pinned = torch.zeros(12 * n, dtype=torch.uint8).pin_memory()
    _abi.check(_abi.lib().rl_map_encode(m.handle, 0, C.c_void_p(pinned.data_ptr()), None))
    assert np.array_equal(pinned.numpy(), raw)


def test_many_threads(cuda):
    maps = [_map(120000 + k, k) for k in range(7)]
    bad = []

    def run(k):
        m, color = maps[k]
        for _ in range(5):
            if not np.array_equal(m.encode(0), np.frombuffer(color.tobytes(), np.uint8)):
                bad.append(k)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(7)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad

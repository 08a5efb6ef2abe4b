"""Two host threads in the library at once, each with its own modules, stream and buffers, on blocks whose
kernels are the same but need different amounts of shared memory: every result has the bits of the same call
made alone."""
import threading

import pytest
import torch

from cssm_b200 import GatedCSSM, GatedDeltaNetCSSM, device_error

pytestmark = pytest.mark.gpu
SHAPES = [(2, 3, 9, 11, 16), (1, 2, 40, 37, 32), (1, 2, 14, 14, 256), (2, 2, 30, 44, 12), (1, 3, 14, 14, 32), (1, 2, 56, 50, 8)]


def _modules(shape):
    C = shape[-1]
    for m in (GatedCSSM(channels=C, kernel_size=1, gate_type="factored"),
              GatedDeltaNetCSSM(channels=C, kernel_size=1, gate_type="factored", delta_key_dim=2)):
        yield m, m.init(7, shape, bias_scale=0.1)


def test_two_threads_give_the_bits_of_one():
    xs = {s: torch.randn(s, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i, s in enumerate(SHAPES)}
    want = {s: [m.bind(v)(xs[s]).clone() for m, v in _modules(s)] for s in SHAPES}
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(2)

    def work(order):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                bound = {s: [m.bind(v) for m, v in _modules(s)] for s in order}
                start.wait(60)
                for _ in range(4):
                    for s in order:
                        got = [b(xs[s]) for b in bound[s]]
                        torch.cuda.current_stream().synchronize()
                        wrong.extend(s for g, w in zip(got, want[s]) if not torch.equal(g, w))
        except Exception as e:                       # a failing launch raises here
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(o,)) for o in (SHAPES, SHAPES[::-1])]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not wrong and not any(t.is_alive() for t in threads), wrong
    assert device_error() == 0

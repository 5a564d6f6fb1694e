"""Other Python threads run while a call of the library waits for room in the stream's queue."""
import importlib.util
import os
import threading
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _encoder():
    spec = importlib.util.spec_from_file_location("sfb_encoder", os.path.join(ROOT, "sf-bert_b200", "encoder.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("what", ["rowdot", "encoder_layer"])
def test_a_full_queue_does_not_stop_other_threads(sfb, what):
    """The stream is given about 1.5 s of work and then more launches than its queue holds, so that the calling thread has to
    wait.  Another thread that wakes every 5 ms meanwhile must not be kept from running for as long as that."""
    lay = sfb.BlockLayout.generate(sfb.LAYOUT_FULL, 1, 2, 64)
    a = torch.randn(4, 64, device="cuda")
    w = _encoder().EncoderLayerWeights(64, 128, torch.bfloat16)
    x = torch.randn(128, 64, device="cuda").to(torch.bfloat16)
    call, n = (lambda: sfb.rowdot(a, a), 4000) if what == "rowdot" else (lambda: sfb.encoder_layer_tensor(x, w, lay, 1, "post", 0.125), 600)
    call()
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def ticker():
        last = time.monotonic()
        while not stop.is_set():
            time.sleep(0.005)
            now = time.monotonic()
            gaps.append(now - last)
            last = now

    t = threading.Thread(target=ticker)
    t.start()
    torch.cuda._sleep(int(1.5 * 1.9e9))                      # a kernel that counts clock cycles
    began = time.monotonic()
    for _ in range(n):
        call()
    issued = time.monotonic() - began
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert issued > 0.7, "the queue took every launch: nothing was waited for"
    assert max(gaps) < 0.5 * issued

"""The argument checks of the operators' C++ host side, without a GPU.  Every call runs in a process of its own, which has to
come back with the exception: a division by zero in C++ would end it with a signal instead."""
import json
import os
import subprocess
import sys

import pytest

pytest.importorskip("torch")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DIVIDE = [
    "sfb.rowdot(torch.zeros(3, 0), torch.zeros(3, 0))",
    "sfb.linear(torch.zeros(3, 0), torch.zeros(0, 16))",
    "sfb.linear(torch.zeros(3, 0), torch.zeros(0, 16), out=torch.zeros(3, 16))",
    "sfb.linear_nt(torch.zeros(3, 0), torch.zeros(16, 0))",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), w, lay(), 0, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), w, lay(nb=0), 1, 'post', 0.125)",
    "sfb.fused_attention(*[torch.zeros(1, 256, 1, 0)] * 3, lay(), out=torch.zeros(1, 256, 1, 0))",
]
REFUSE = [
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), w, lay(), -1, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), w, lay(), 3, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(255, 64), w, lay(), 1, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(1, 256, 64), w, lay(), 1, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), layer(w1=torch.zeros(64, 128, 1)), lay(), 1, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), layer(wo=torch.zeros(64, 64, 1)), lay(), 1, 'post', 0.125)",
    "sfb.encoder_layer_tensor(torch.zeros(256, 64), layer(w2=torch.zeros(128)), lay(), 1, 'post', 0.125)",
    "sfb.linear(torch.zeros(2, 64), torch.zeros(64, 32, 1))",
    "sfb.linear(torch.zeros(2, 64), torch.zeros(64))",
    "sfb.linear_nt(torch.zeros(2, 64), torch.zeros(32, 64, 1))",
]

# one child that loads the package once and forks for every call
RUNNER = """
import json, os, sys, types
sys.path.insert(0, %r)
import torch
import __graft_entry__ as ge
sfb = ge.load_package()
def lay(nb=4, bs=64):
    return types.SimpleNamespace(heads=1, nb=nb, block_size=bs, blocks=nb, nn_max=1, nn_lut=None, mask_np=None)
def layer(**changed):
    z = torch.zeros
    w = dict(fused_qkv=lambda: (z(64, 192), z(192)), wo=z(64, 64), w1=z(64, 128), w2=z(128, 64), b1=z(128))
    w.update({n: z(64) for n in ("bo", "b2", "g1", "g2", "be1", "be2")})
    w.update(changed)
    return types.SimpleNamespace(**w)
w = types.SimpleNamespace()
for call in json.load(sys.stdin):
    r, wr = os.pipe()
    pid = os.fork()
    if pid == 0:
        try:
            eval(call)
            said = "returned"
        except Exception as e:
            said = type(e).__name__
        os.write(wr, said.encode())
        os._exit(0)
    os.close(wr)
    said = os.read(r, 100).decode()
    status = os.waitpid(pid, 0)[1]
    print(json.dumps([call, said if status == 0 else "ended with status %%d" %% status]), flush=True)
""" % ROOT


@pytest.fixture(scope="module")
def said():
    r = subprocess.run([sys.executable, "-c", RUNNER], input=json.dumps(DIVIDE + REFUSE), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-1000:]
    return dict(json.loads(line) for line in r.stdout.splitlines())


@pytest.mark.parametrize("call", DIVIDE)
def test_sizes_of_zero_that_something_is_divided_by(said, call):
    assert said[call] == "ZeroDivisionError"


@pytest.mark.parametrize("call", REFUSE)
def test_shapes_that_do_not_fit(said, call):
    assert said[call] == "AssertionError"

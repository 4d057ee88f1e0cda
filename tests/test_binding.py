"""The compiled way to the op launches (csrc/binding.cpp) against the Python way behind it: the same results, the same refusals."""
import importlib

import numpy as np
import pytest
import torch

from inferi_b200 import ops, quant
from inferi_b200.ops import AttnParams, FusedAttention, GemmQuant, GemvQuant, GpuQuantTensor, InferiError, RmsNorm, RmsNormConfig, RoPE, RoPEConfig, Sampler, Silu


class PythonOnly:
    """Takes no call"""
    gemv = gemm = rms_norm = rope = silu = add = attention = argmax = sample = staticmethod(lambda *a: -1)


class Recorded:
    """The compiled binding, and what its entries answered: name -> statuses"""
    def __init__(self):
        self.binding, self.answers = importlib.import_module("inferi_b200._binding"), {}

    def __getattr__(self, name):
        entry = getattr(self.binding, name)

        def call(*args):
            rc = entry(*args)
            self.answers.setdefault(name, []).append(rc)
            return rc
        return call


ENTRIES = {"gemv", "gemm", "rms_norm", "rope", "silu", "add", "attention", "argmax", "sample"}


class Tagged(torch.Tensor):
    pass


def test_the_binding_takes_nothing_that_it_cannot_check():
    """Not tensors, tensors of the host, wrong counts and closed handles are left to the Python way, and leave no error behind."""
    binding = pytest.importorskip("inferi_b200._binding")
    t = torch.zeros(8)
    for args in [(1, t, 1, 8, 8, t), (None, t, 1, 8, 8, t), (1, None, 1, 8, 8, "x"), (1, t), ()]:
        assert binding.gemv(*args) == binding.gemm(*args) == -1
    assert binding.rms_norm(1, t, t, t, 1e-5) == binding.rms_norm(1, t, t, t, None) == -1
    assert binding.rope(1, 0, t, t, 8, 8, 2**40, 1e4) == binding.rope(1, 0, t, t, -1, 8, 0, 1e4) == -1
    assert binding.silu(1, t, t) == binding.add(0, t, t) == binding.argmax(1, t, t) == binding.sample(1, t, 8, 1.0, 0.9, 0.5, t) == -1
    assert binding.attention(1, b"x" * 24, t, t, t, t) == binding.attention(1, 7, t, t, t, t) == -1


def calls(b, dev, wrap=lambda t: t):
    """name -> a launch that returns what it wrote; inputs are the same every time"""
    g = torch.Generator(device=dev).manual_seed(3)

    def rand(*shape, dtype=torch.float32):
        return wrap(torch.randn(*shape, generator=g, device=dev).to(dtype))

    m = GpuQuantTensor(b, quant.Q4_K, 256, 512, quant.random_blocks(quant.Q4_K, 256, 512, seed=1))
    # views into larger tensors: 256-byte aligned rows with an offset
    x, y, w = rand(4, 512)[1], rand(512), rand(512)
    X = rand(9, 512)
    kv = {d: (rand(64, 128, dtype=d), rand(64, 128, dtype=d)) for d in (torch.float16, torch.float32)}
    q = rand(256)

    def new(*shape, dtype=torch.float32):
        return wrap(torch.zeros(*shape, device=dev, dtype=dtype))

    def gemv():
        out = new(256); GemvQuant(b).launch(out, m, x); return out

    def gemm():
        out = new(9, 256); GemmQuant(b).launch(out, m, X); return out

    def rms():
        out = new(512); RmsNorm(b).launch(RmsNormConfig(1e-5), out, x, w); return out

    def rope():
        a, k = q.clone(), q[:128].clone(); RoPE(b).launch(0, RoPEConfig(64, 128, 7, 5e5), a, k); return torch.cat([a, k])

    def rope_of_another_model():
        a, k = q.clone(), q[:128].clone(); RoPE(b).launch(1, RoPEConfig(128, 128, 7, 1e4), a, k); return torch.cat([a, k])

    def silu():
        a = x.clone(); Silu(b).launch(a, y); return a

    def add():
        a = x.clone(); ops.add_assign(b, a, y); return a

    def attention(dtype):
        out = new(256); FusedAttention(b).launch(AttnParams(64, 128, 2, 4, 64, 40), q, *kv[dtype], out); return out

    def argmax():
        out = new(1, dtype=torch.int32); ops.argmax(b, y, out); return out

    def sample():
        return Sampler(b, 512, 0.8, 0.9).sample(y, 0.4)

    return dict(gemv=gemv, gemm=gemm, rms=rms, rope=rope, rope2=rope_of_another_model, rope_again=rope, silu=silu, add=add, attention_f16=lambda: attention(torch.float16),
                attention_f32=lambda: attention(torch.float32), argmax=argmax, sample=sample)


@pytest.mark.gpu
def test_both_ways_launch_the_same(backend, monkeypatch):
    """Bit for bit, on the default stream and on another one, with plain tensors (which the binding takes: every entry launches) and with a subclass
    (which takes the Python way)"""
    recorded = Recorded()
    assert ops._fast is recorded.binding
    monkeypatch.setattr(ops, "_fast", recorded)
    fast = {n: f().cpu() for n, f in calls(backend, "cuda").items()}
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        aside = {n: f() for n, f in calls(backend, "cuda").items()}
    side.synchronize()
    assert {n: set(rc) for n, rc in recorded.answers.items()} == {n: {0} for n in ENTRIES}
    recorded.answers.clear()
    tagged = {n: f().cpu().as_subclass(torch.Tensor) for n, f in calls(backend, "cuda", lambda t: t.as_subclass(Tagged)).items()}
    assert {n: set(rc) for n, rc in recorded.answers.items()} == {n: {-1} for n in ENTRIES}
    monkeypatch.setattr(ops, "_fast", PythonOnly)
    slow = {n: f().cpu() for n, f in calls(backend, "cuda").items()}
    for n in fast:
        assert torch.equal(fast[n], slow[n]) and torch.equal(aside[n].cpu(), slow[n]) and torch.equal(tagged[n], slow[n]), n


@pytest.mark.gpu
def test_both_ways_refuse_the_same(backend, monkeypatch):
    b, c = backend, lambda *s, **k: torch.zeros(*s, device="cuda", **k)
    m = GpuQuantTensor(b, quant.Q4_K, 256, 512, quant.random_blocks(quant.Q4_K, 256, 512, seed=1))
    closed = GpuQuantTensor(b, quant.Q4_K, 256, 512, quant.random_blocks(quant.Q4_K, 256, 512, seed=1))
    closed.close()
    p = AttnParams(64, 128, 2, 4, 64, 40)
    refused = [
        lambda: GemvQuant(b).launch(c(256), m, c(511)), lambda: GemvQuant(b).launch(c(256), m, c(512, dtype=torch.float64)), lambda: GemvQuant(b).launch(c(256), m, c(1024)[::2]),
        lambda: GemvQuant(b).launch(c(256), m, torch.zeros(512)), lambda: GemvQuant(b).launch(c(256), m, c(513)[1:]), lambda: GemvQuant(b).launch(c(256), closed, c(512)),
        lambda: GemmQuant(b).launch(c(2, 256), m, c(2, 511)), lambda: GemmQuant(b).launch(c(3, 256), m, c(2, 512)), lambda: GemmQuant(b).launch(c(256), m, c(512)),
        lambda: RmsNorm(b).launch(RmsNormConfig(1e-5), c(8), c(8), c(9)), lambda: RmsNorm(b).launch(RmsNormConfig(1e-5), c(0), c(0), c(0)),
        lambda: RoPE(b).launch(0, RoPEConfig(64, 128, 0, 1e4), c(256), c(64)), lambda: RoPE(b).launch(5, RoPEConfig(64, 128, 0, 1e4), c(256), c(128)),
        lambda: Silu(b).launch(c(8), c(9)), lambda: ops.add_assign(b, c(8), c(9)), lambda: ops.argmax(b, c(8), c(1, dtype=torch.int64)), lambda: ops.argmax(b, c(0), c(1)),
        lambda: FusedAttention(b).launch(p, c(256), c(64, 128), c(64, 128, dtype=torch.float16), c(256)), lambda: FusedAttention(b).launch(p, c(256), c(63, 128), c(64, 128), c(256)),
        lambda: FusedAttention(b).launch(p, c(255), c(64, 128), c(64, 128), c(256)), lambda: FusedAttention(b).launch(AttnParams(64, 128, 2, 4, 64, 64), c(256), c(64, 128), c(64, 128), c(256)),
        lambda: Sampler(b, 8, 1.0, 0.9).sample(c(9), 0.5), lambda: Sampler(b, 8, 1.0, 0.9).sample(c(8), 1.0), lambda: RmsNorm(None).launch(RmsNormConfig(1e-5), torch.zeros(4), c(4), c(4)),
    ]

    def answers():
        out = []
        for f in refused:
            with pytest.raises((InferiError, ValueError)) as e:
                f()
            out.append((type(e.value), str(e.value)))
        return out

    assert ops._fast is importlib.import_module("inferi_b200._binding")
    fast = answers()
    monkeypatch.setattr(ops, "_fast", PythonOnly)
    assert answers() == fast

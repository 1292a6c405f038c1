"""The benchmark's step is the engine's step, on the CPU with the library calls recorded,
and the net kernel it names is the one the library's rule takes."""
import pytest

import bench


@pytest.mark.parametrize("method,widths", [("fd", (64, 64)), ("adjoint", (64, 64)), ("adjoint", (128, 128)),
                                           ("fd_split", (64, 64))])
def test_bench_step_issues_the_engine_s_calls(monkeypatch, method, widths):
    from amlp import engine
    from amlp.configs import make_state
    calls = []
    monkeypatch.setattr(engine, "call", lambda name, *args: calls.append(name))
    monkeypatch.setattr(engine, "size_query", lambda *args: 64)
    monkeypatch.setattr(engine, "_stream", lambda: 0)
    monkeypatch.setattr(engine._lib, "check_device", lambda: None)
    net = engine.EnergyNet.xavier(47, widths, "tanh", 1, "cpu")
    s = engine.System(make_state(27, "cube26", 0.3, seed=1), "cube26", engine.Hypers(), net, 1.0, 0.005, device="cpu")
    calls.clear()
    s._step_kernels(method)
    own, events = list(calls), []
    calls.clear()
    launched = bench.engine_step(s, method, lambda: events.append(len(calls)), lambda: events.append(len(calls)))
    assert calls == own
    assert events == [1, len(own) - 1]  # around the force pass alone
    assert launched == sum(bench.LAUNCHES[c] for c in own)
    assert s.timestep == 1


@pytest.mark.parametrize("D,widths,act,kernel", [
    (47, (150,) * 4, "relu", "k_mlp_pair"), (121, (150,) * 4, "relu", "k_mlp_pair"),
    (47, (128, 128), "silu", "k_mlp_pair"), (47, (64,) * 3, "tanh", "k_mlp_pair"),
    (47, (128,) * 3, "silu", "k_mlp_grad"), (47, (96,) * 3, "tanh", "k_mlp_grad"),
    (47, (160,) * 2, "silu", "k_mlp_grad")])
def test_net_kernel_of_the_wide_path(D, widths, act, kernel):
    assert bench.net_kernel(D, widths, act) == kernel

"""Calls on a NeuralSDF after its state has changed under it: a captured
training step must not outlive the points and the input map it was made for,
and a wait that ran out must not go unreported."""
import ctypes

import numpy as np
import pytest
import torch

import rayengine_b200 as rb

pytestmark = pytest.mark.gpu

BOX = ([-40.0, -6.0, -20.0], [40.0, 11.0, 60.0])
OTHER = ([-20.0, -5.0, -10.0], [30.0, 9.0, 50.0])


def _generate(net, points):
    t = rb.configs.TerrainConfig(width=64, height=36)
    net.generate(t.params(), t.camera(), t.width, t.height, points, seed=4)


def _captured(points, steps=(8, 2)):
    """A model whose captured step has room left in its loss history (the
    first call allocates 8 entries, the second grows them to 16)."""
    net = rb.NeuralSDF(*BOX, 0.5, 3)
    _generate(net, points)
    for n in steps:
        net.train(n, batch=512)
    return net


@pytest.mark.parametrize("points", [700, 40000])
def test_train_after_generate(cuda, tmp_path, points):
    with _captured(5000) as net, rb.NeuralSDF(*BOX, 0.5, 3) as fresh:
        ck = str(tmp_path / "state.rnsdf")
        net.save(ck)
        fresh.load(ck)
        for m in (net, fresh):
            _generate(m, points)
        assert np.array_equal(net.train(4, batch=512), fresh.train(4, batch=512))
        assert np.array_equal(net.get_params(), fresh.get_params())


def test_train_after_load(cuda, tmp_path):
    ck = str(tmp_path / "other.rnsdf")
    with rb.NeuralSDF(*OTHER, 0.7, 3) as other:
        _generate(other, 5000)
        other.train(10, batch=512)
        other.save(ck)
    with _captured(5000) as net, rb.NeuralSDF(*BOX, 0.5, 3) as fresh:
        _generate(fresh, 5000)
        for m in (net, fresh):
            m.load(ck)
        assert np.array_equal(net.train(4, batch=512), fresh.train(4, batch=512))
        assert np.array_equal(net.get_params(), fresh.get_params())


@pytest.mark.parametrize("thread", [0, 1, 127, 128, 600, 1023, 1024])
def test_any_threads_failed_wait_is_reported(cuda, thread):
    """The evaluation kernel's 1024 threads wait each for itself: one whose
    wait ran out (1024: none) is reported, whichever row it holds."""
    with rb.NeuralSDF(*BOX, 0.5, 3) as net:
        got = ctypes.c_int(-1)
        rb.api.call("re_nsdf_check_report", net._h, thread, ctypes.byref(got))
        assert got.value == (1 if thread < 1024 else 0)


def test_loss_gradient_refuses_host_memory(cuda):
    with rb.NeuralSDF(*BOX, 0.5, 3) as net:
        _generate(net, 512)
        xyzl = torch.from_numpy(net.data(512)).cuda()
        want, _ = net.loss_grad(xyzl)
        host = np.zeros(net.num_params, np.float32)
        with pytest.raises(rb.RayEngineError) as e:
            rb.api.call("re_nsdf_loss_grad", net._h, xyzl.data_ptr(), 512, host.ctypes.data, None,
                        None)
        assert e.value.status == 1 and not host.any()
        pinned = torch.zeros(net.num_params).pin_memory()  # the device reaches it
        rb.api.call("re_nsdf_loss_grad", net._h, xyzl.data_ptr(), 512, pinned.data_ptr(), None,
                    None)
        assert torch.equal(pinned, want.cpu())

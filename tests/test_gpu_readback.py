"""The gradient read-back: transposed on the device, in chunks, to the reference's file order."""
import numpy as np
import pytest

import denise_b200 as dn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(33, 20), (1, 40), (1201, 1801)])
@pytest.mark.parametrize("acc", ["f32", "f64"])
def test_gradient_readback_order(nx, ny, acc):
    """Read-back in chunks (the largest case needs two a field): every element in its place."""
    from denise_b200 import _lib, synth

    p = synth.c0_params(nx=nx, ny=ny, nt=10, fw=0, store_snapshots=1,
                        grad_accum=_lib.ACC_F64 if acc == "f64" else _lib.ACC_F32)
    one = np.ones((nx, ny), np.float32)
    m = dn.Model(p, 3000 * one, 1700 * one, 2000 * one)
    rng = np.random.default_rng(nx)
    g = [rng.standard_normal((nx, ny)).astype(np.float32) for _ in range(3)]
    m.set_gradient(*g)
    for a, b in zip(m.gradient(), g):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("acc", ["f32", "f64"])
@pytest.mark.parametrize("nx,ny", [(64, 64), (241, 17), (300, 150), (1201, 1801), (33, 200)])
def test_readback_takes_no_more_memory_than_the_gradient(nx, ny, acc):
    """The first read-back of a gradient costs what that gradient needs, not the largest chunks; sizes
    on both sides of the line to the single copy, and larger and smaller ones in turn."""
    from denise_b200 import _lib, synth

    p = synth.c0_params(nx=nx, ny=ny, nt=10, fw=0, store_snapshots=1,
                        grad_accum=_lib.ACC_F64 if acc == "f64" else _lib.ACC_F32)
    one = np.ones((nx, ny), np.float32)
    m = dn.Model(p, 3000 * one, 1700 * one, 2000 * one)
    rng = np.random.default_rng(ny)
    g = [rng.standard_normal((nx, ny)).astype(np.float32) for _ in range(3)]
    m.set_gradient(*g)
    m.gradient()
    dn.device_trim(0)
    free = dn.device_memory(0)[0]
    got = m.gradient()
    taken = free - dn.device_memory(0)[0]
    assert taken <= 2 * min(4 * nx * ny, 8 << 20) + (4 << 20), taken   # two chunks, in the driver's 2 MB steps
    for a, b in zip(got, g):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("idle", [False, True])
def test_gradient_readback_on_a_full_device(idle):
    """No device memory left for the read-back's chunks: the gradient still comes out, by the
    blocks that the library keeps idle (idle) or without any device memory."""
    import torch

    from denise_b200 import _lib, synth

    p = synth.c0_params(nx=1201, ny=1801, nt=10, fw=0, store_snapshots=1, grad_accum=_lib.ACC_F64)
    one = np.ones((p.nx, p.ny), np.float32)
    m = dn.Model(p, 3000 * one, 1700 * one, 2000 * one)
    rng = np.random.default_rng(3)
    g = [rng.standard_normal((p.nx, p.ny)).astype(np.float32) for _ in range(3)]
    m.set_gradient(*g)
    m.gradient()   # its kernels are loaded before the device is full
    dn.device_trim(0)
    if idle:
        dn.Model(p, 3000 * one, 1700 * one, 2000 * one).close()
    full, size = [], 64 << 30
    while size >= 1 << 20:
        try:
            full.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    try:
        assert torch.cuda.mem_get_info(0)[0] < 8 << 20   # a chunk does not fit
        got = m.gradient()
    finally:
        full.clear()
        torch.cuda.empty_cache()
    for a, b in zip(got, g):
        np.testing.assert_array_equal(a, b)

"""The training kernels at the edges of their tiles: one row, one short of a
128-row tile, one past it, and more tiles than a pass over the device's SMs
holds; and inputs whose addresses allow no 16-byte loads."""
import ctypes as C

import numpy as np
import pytest

from avbd_b200 import abi, learned
from avbd_b200.solver import load_library

pytestmark = pytest.mark.gpu


def _case(B):
    rng = np.random.default_rng(B)
    p = learned.init_params(seed=B)
    p[learned.HID * learned.DIN:learned.HID * learned.DIN + learned.HID] = rng.normal(0, 0.1, learned.HID)
    norm = np.ones(learned.NNORM, np.float32)
    norm[:learned.DIN] = rng.normal(0, 0.1, learned.DIN)
    norm[learned.YM:learned.YM + learned.USED] = rng.normal(0, 0.1, learned.USED)
    X = rng.normal(size=(B, learned.DIN)).astype(np.float32)
    T = rng.normal(size=(B, learned.USED)).astype(np.float32)
    return p, norm, X, T


# 5e-3: the bar of the oracle comparison at ordinary batches (a different fp32
# accumulation order moves single BF16 roundings of the activations)
@pytest.mark.parametrize("B", [1, 127, 128, 129, 148 * 128 + 37])
def test_gradients_at_tile_edges(cuda_lib, oracle_lib, B):
    from oracle import mlp_oracle as M
    p, norm, X, T = _case(B)
    loss, g = learned.gradients(p, norm, X, T)
    want_loss, want = M.forward_backward(p, norm, X, T, rounded=True)
    assert abs(loss - want_loss) <= 1e-4 * max(1.0, abs(want_loss))
    for a, b in ((M.OW1, M.OB1), (M.OB1, M.OW2), (M.OW2, M.OB2), (M.OB2, M.OW3), (M.OW3, M.OB3), (M.OB3, M.OW4),
                 (M.OW4, M.OB4), (M.OB4, M.NPARAM)):
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 5e-3 * max(np.linalg.norm(want[a:b]), 1e-12)


def test_gradients_of_unaligned_inputs(cuda_lib):
    """Parameters, features and targets four bytes off a 16-byte boundary give
    the aligned call's gradients bit for bit."""
    import torch
    lib = load_library()
    p, norm, X, T = _case(200)
    want_loss, want = learned.gradients(p, norm, X, T)

    def shifted(a):
        t = torch.zeros(a.size + 1, dtype=torch.float32, device="cuda")
        t[1:] = torch.from_numpy(a.ravel()).cuda()
        return t[1:]

    args = [shifted(a) for a in (p, norm, X, T)]
    grad = torch.zeros(learned.NPARAM, device="cuda")
    loss = torch.zeros(1, device="cuda")
    ws = torch.empty(lib.avbd_mlp_workspace_bytes(200), dtype=torch.uint8, device="cuda")
    rc = lib.avbd_mlp_gradients(*(a.data_ptr() for a in args), 200, ws.data_ptr(), grad.data_ptr(), loss.data_ptr(),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert float(loss.item()) == want_loss
    assert np.array_equal(grad.cpu().numpy(), want)


def _device_step(B):
    """(tensors, arguments of a training step up to the step number) of a fresh network."""
    import torch
    p, norm, X, T = _case(B)
    t = {"prm": p, "norm": norm, "x": X, "t": T, "m": np.zeros_like(p), "v": np.zeros_like(p)}
    t = {k: torch.from_numpy(np.ascontiguousarray(v, np.float32)).cuda() for k, v in t.items()}
    # a workspace with another step's partial gradients in it
    t["ws"] = torch.ones(load_library().avbd_mlp_workspace_bytes(B) // 4, dtype=torch.float32, device="cuda")
    t["loss"] = torch.full((1,), 7.0, device="cuda")
    return t, [t[k].data_ptr() for k in ("prm", "norm", "x", "t")] + [B] + [t[k].data_ptr() for k in ("m", "v")]


@pytest.mark.parametrize("B", [100, 1000])
def test_step_whose_wait_gave_up_changes_nothing(cuda_lib, B):
    import torch
    lib = load_library()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    t, args = _device_step(B)
    before = t["prm"].clone()
    tail = (C.c_float(1e-2), t["ws"].data_ptr(), t["loss"].data_ptr(), stream)
    assert lib.avbd_mlp_train_step_wait_timeout_for_testing(*args, 1, *tail) == 0
    assert lib.avbd_mlp_workspace_status(t["ws"].data_ptr(), B, stream) == abi.ERR_RUNTIME_FAILURE
    assert torch.equal(t["prm"], before) and not t["m"].any() and not t["v"].any()
    assert float(t["loss"]) == 7.0
    # the device and the workspace are as good as new
    assert lib.avbd_mlp_train_step(*args, 1, *tail) == 0
    assert lib.avbd_mlp_workspace_status(t["ws"].data_ptr(), B, stream) == 0
    fresh, fresh_args = _device_step(B)
    assert lib.avbd_mlp_train_step(*fresh_args, 1, C.c_float(1e-2), fresh["ws"].data_ptr(), fresh["loss"].data_ptr(),
                                   stream) == 0
    assert all(torch.equal(t[k], fresh[k]) for k in ("prm", "m", "v", "loss"))
    assert not torch.equal(t["prm"], before)


def test_inference_keeps_a_shared_workspaces_training_status(cuda_lib):
    import torch
    lib, B = load_library(), 1000
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    t, args = _device_step(B)
    tail = (C.c_float(1e-2), t["ws"].data_ptr(), t["loss"].data_ptr(), stream)
    assert lib.avbd_mlp_train_step_wait_timeout_for_testing(*args, 1, *tail) == 0
    out = torch.zeros(B, learned.USED, device="cuda")
    assert lib.avbd_mlp_infer(*(t[k].data_ptr() for k in ("prm", "norm", "x")), B, out.data_ptr(), t["ws"].data_ptr(),
                              stream) == 0
    assert lib.avbd_mlp_workspace_status(t["ws"].data_ptr(), B, stream) == abi.ERR_RUNTIME_FAILURE

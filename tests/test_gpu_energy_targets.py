"""Gradients of the penetration energy with morph targets around the eight that
the skin adjoint sums at once, against the FP64 reference of oracle/energy.py
on the GPU's own colliding pairs (bounds as test_gpu_energy.py)."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300.energy import penetration_energy
from test_gpu_energy import E_RTOL, GRAD_RTOL, leaf, make, pair_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_targets", [1, 7, 8, 9, 17])
def test_target_counts(gpu_ctx, port, n_targets):
    sc, col, problem, fid = make(gpu_ctx, port, n_meshes=4, rings=30, around=20, n_targets=n_targets, grid=100)
    aa, mw = leaf(sc.axis_angles), leaf(sc.morph_weights)
    E = penetration_energy(aa, mw, col)
    E.backward()
    pairs = pair_array(col)
    assert len(pairs) > 0
    e64, ga64, gw64 = problem(pairs).value_and_grad(aa.detach().cpu().double().numpy(),
                                                    mw.detach().cpu().double().numpy())
    assert abs(E.item() - e64) <= E_RTOL * e64
    for got, want in ((aa.grad, ga64), (mw.grad, gw64)):
        assert np.linalg.norm(got.cpu().double().numpy() - want) <= GRAD_RTOL * np.linalg.norm(want)
    col.close()
    gpu_ctx.free_tree(fid)

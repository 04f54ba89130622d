"""The assembly's gather at the edges of its chunks, on element blocks written by the test.

F tets around a common edge give slots of F contributions (one chunk holds 32), next to slots of one or two; one more
vertex belongs to no tet.  A float32 sum of m terms in any order is within m 2^-24 sum |term| of the exact one.
"""
import numpy as np
import pytest
import torch

from mfem_gb300 import MixedFEMSolver, Model

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def fan(F):
    """F tets (0, 1, rim i, rim i + 1), closed for F >= 3, and the lone vertex F + 3 (F + 4 if open)."""
    closed = F >= 3
    rim = F if closed else F + 1
    ang = 2.0 * np.pi * np.arange(rim) / max(rim, 6 if not closed else rim)
    x = np.concatenate([[[0, 0, -0.5], [0, 0, 0.5]], np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1), [[3.0, 0, 0]]])
    tets = np.array([[0, 1, 2 + i, 2 + (i + 1) % rim] for i in range(F)])
    tets[1::2] = tets[1::2][:, [2, 0, 3, 1]]  # corners of the shared edge in either order
    e = np.swapaxes(x[tets[:, 1:]] - x[tets[:, :1]], 1, 2)
    flip = np.linalg.det(e) < 0
    tets[flip] = tets[flip][:, [0, 2, 1, 3]]
    e = np.swapaxes(x[tets[:, 1:]] - x[tets[:, :1]], 1, 2)
    return x.astype(np.float32), tets.astype(np.int32), np.linalg.inv(e).astype(np.float32)


@pytest.mark.parametrize("F", [1, 2, 5, 16, 31, 32, 33, 40, 65, 97])
def test_gather_of_written_blocks(F):
    x, tets, poses = fan(F)
    n, T = len(x), len(tets)
    mass = np.ones(n, np.float32)
    model = Model(x, np.zeros_like(x), mass, mass, tets, poses, np.tile(np.float32([1e4, 1e4, 0.0]), (T, 1)),
                  (0.0, 0.0, 0.0), device=DEV)
    solver = MixedFEMSolver(model, iterations=1, energy="arap")
    q, dt = torch.as_tensor(x, device=DEV), 1.0 / 64.0
    solver.predict(q, torch.zeros_like(q), dt)
    solver.update_system(q)
    rng = np.random.default_rng(F)
    ke = rng.normal(0.0, 1.0, (T, 10, 3, 3)).astype(np.float32)
    fe = rng.normal(0.0, 1.0, (T, 4, 3)).astype(np.float32)
    for name, a in (("element_hessian", ke), ("element_rhs", fe)):
        solver.write_buffer(name, torch.as_tensor(a).reshape(-1))
    for name, a in (("element_hessian", ke), ("element_rhs", fe)):
        np.testing.assert_array_equal(solver.read_buffer(name).cpu().numpy(), a.reshape(-1))
    solver.assemble(q, dt)

    def dense(blocks):
        H, m = np.zeros((n, n, 3, 3)), np.zeros((n, n, 1, 1))
        for e in range(T):
            b = 0
            for k in range(4):
                for l in range(k, 4):
                    i, j = tets[e, k], tets[e, l]
                    H[i, j] += blocks[e, b]
                    m[i, j] += 1
                    if k != l:
                        H[j, i] += blocks[e, b].T
                        m[j, i] += 1
                    b += 1
        return H, m

    H, m = dense(ke.astype(np.float64))
    A, _ = dense(np.abs(ke.astype(np.float64)))
    diag = np.arange(n)
    H[diag, diag] += np.eye(3) / dt ** 2
    A[diag, diag] += np.eye(3) / dt ** 2
    rp, ci = (solver.read_buffer(k).cpu().numpy() for k in ("row_ptr", "col_idx"))
    vals = solver.read_buffer("h_values").cpu().numpy().reshape(-1, 3, 3)
    got, seen = np.zeros((n, n, 3, 3), np.float32), np.zeros((n, n), bool)
    for i in range(n):
        got[i, ci[rp[i]:rp[i + 1]]] = vals[rp[i]:rp[i + 1]]
        seen[i, ci[rp[i]:rp[i + 1]]] = True
    assert not np.abs(H[~seen]).any()
    assert np.all(np.abs(got - H) <= (m + 2) * 2.0 ** -24 * A)
    off = ~np.eye(n, dtype=bool)
    np.testing.assert_array_equal(got[off], np.swapaxes(got, 0, 1).swapaxes(2, 3)[off])

    # rest pose, at rest: g is the sum of the right-hand sides
    g, ag, mg = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros((n, 1))
    for k in range(4):
        np.add.at(g, tets[:, k], fe[:, k].astype(np.float64))
        np.add.at(ag, tets[:, k], np.abs(fe[:, k]).astype(np.float64))
        np.add.at(mg, tets[:, k], 1)
    rhs = solver.read_buffer("rhs").cpu().numpy().reshape(n, 3)
    assert np.all(np.abs(rhs - g) <= mg * 2.0 ** -24 * ag)
    det = np.linalg.det(got[diag, diag].astype(np.float64))
    inv = solver.read_buffer("precond").cpu().numpy().reshape(-1, 3, 3)[:n]
    ref = np.linalg.inv(got[diag, diag].astype(np.float64))
    assert np.all(np.abs(det) > 1.0)  # diagonally dominant: 4096 against sums of F unit normals
    np.testing.assert_allclose(inv, ref, rtol=0, atol=1e-5 * np.abs(ref).max())

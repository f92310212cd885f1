"""The two-stage eigensolver at the edges of its tiles: padded sizes around
multiples of 16 and the shared-memory limit, numbers of vectors around the
back-transform's groups, and matrices whose reflectors vanish (diagonal, banded,
block diagonal, zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(96, 8, "dense"), (97, 3, "banded"), (112, 33, "blocks"), (113, 9, "diagonal"), (128, 20, "dense"),
         (153, 2, "dense"), (154, 1, "dense"), (160, 7, "dense"), (161, 8, "banded"), (175, 9, "dense"), (176, 16, "blocks"),
         (177, 17, "diagonal"), (200, 31, "dense"), (256, 32, "banded"), (273, 33, "dense"), (289, 5, "blocks"),
         (300, 40, "diagonal"), (400, 3, "dense"), (416, 24, "dense"), (417, 24, "dense"), (433, 65, "blocks"),
         (160, 12, "zero"), (818, 6, "banded"), (180, 180, "dense")]


def _matrix(rng, n, kind):
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A = (A + A.conj().T) / 2
    i = np.arange(n)
    if kind == "diagonal":  # with repeated values
        return np.diag(np.round(4 * rng.standard_normal(n)) / 4).astype(complex)
    if kind == "zero":
        return np.zeros((n, n), complex)
    if kind == "banded":
        A[np.abs(i[:, None] - i[None, :]) > 3] = 0.0
    if kind == "blocks":
        b = i // 37
        A[b[:, None] != b[None, :]] = 0.0
    return A


@pytest.mark.parametrize("n,nev,kind", CASES)
def test_two_stage_edges(ctx, n, nev, kind):
    rng = np.random.default_rng(1000 + n)
    A = np.stack([_matrix(rng, n, kind) for _ in range(2)])
    w, Z = ctx.heev(A, nev)
    for b in range(2):
        full = np.linalg.eigvalsh(A[b])
        scale = max(np.max(np.abs(full)), 1.0)
        assert np.max(np.abs(w[b] - full[:nev])) < 1e-12 * scale * n
        R = A[b] @ Z[b] - Z[b] * w[b]
        assert np.max(np.linalg.norm(R, axis=0)) < 1e-10 * scale
        assert np.max(np.abs(Z[b].conj().T @ Z[b] - np.eye(nev))) < 1e-10


@pytest.mark.parametrize("n,nev", [(96, 8), (113, 9), (129, 16), (160, 5)])
def test_many_small_matrices(ctx, n, nev):
    """More small matrices than SMs: two CTAs per SM in both reduction stages."""
    rng = np.random.default_rng(n)
    A = np.stack([_matrix(rng, n, ("dense", "banded", "blocks", "diagonal")[b % 4]) for b in range(151)])
    w, Z = ctx.heev(A, nev)
    for b in (0, 1, 2, 3, 75, 147, 148, 149, 150):
        full = np.linalg.eigvalsh(A[b])
        scale = max(np.max(np.abs(full)), 1.0)
        assert np.max(np.abs(w[b] - full[:nev])) < 1e-12 * scale * n
        R = A[b] @ Z[b] - Z[b] * w[b]
        assert np.max(np.linalg.norm(R, axis=0)) < 1e-10 * scale
        assert np.max(np.abs(Z[b].conj().T @ Z[b] - np.eye(nev))) < 1e-10

"""Accuracy of FP64 products (default kernel) against extended precision, element by element and entry by entry, for
fields that peak at a vertex, an edge or a face, numerical tails, smooth and random fields, on cubic, stretched, curved
and uneven elements: no further from the exact product than FP64 arithmetic."""
import numpy as np
import pytest

from montjoie_gb300.operator import FemMatrixFreeOperator
from montjoie_gb300.problem import derivative_matrix, gauss_lobatto, local_numbering

pytestmark = pytest.mark.gpu

FP64_PIPE_TILE = {1: 30, 2: 12, 3: 8, 4: 4, 5: 3, 6: 2, 7: 2, 8: 1}
U = 2.0 ** -53


def _matrix(order):
    G = derivative_matrix(gauss_lobatto(order)[0])
    return np.ascontiguousarray(0.5 * (G - G[::-1, ::-1]))


def _factors(order, rng):
    """name -> symmetric factors [i, j, k, (xx, xy, xz, yy, yz, zz)]: quadrature weights times a metric."""
    w, x, n = gauss_lobatto(order)[1], gauss_lobatto(order)[0], order + 1
    W = np.einsum("i,j,k->ijk", w, w, w)

    def make(skew, aspect=(1.0, 1.0, 1.0), uneven=1.0):
        a = np.array(aspect) / np.cbrt(np.prod(aspect))
        B = np.zeros((n, n, n, 6))
        for q, (r, s) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
            B[..., q] = W * uneven / (a[r] * a[s]) * (rng.uniform(1 - skew, 1 + skew, W.shape) if r == s
                                                      else skew * rng.uniform(-1, 1, W.shape))
        return B

    return {"cubic": make(0.02), "skewed": make(0.3), "rectangular": make(0.0), "stretched": make(0.05, (1.0, 8.0, 0.5)),
            "curved": make(0.05, uneven=1 + x[:, None, None] * x[None, :, None]),
            "uneven": make(0.05, uneven=2.0 ** rng.uniform(-9, 0, W.shape))}


def _fields(order, rng):
    n = order + 1
    x = gauss_lobatto(order)[0]
    X, Y, Z = np.meshgrid(x, x, x, indexing="ij")
    i, j, k = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    noise = rng.uniform(-1, 1, X.shape)
    vertex, edge, face, inner = (i + j + k == 0), (i + j == 0), k == 0, j == n // 2
    f = {"random": noise, "smooth": np.sin(1.3 * X + 1) + np.cos(0.7 * Y) * np.sin(1.3 * Z + 0.5),
         "plane wave": np.sin(3 * X + 0.4), "vertex alone": vertex * 1.0, "zero": 0 * X,
         "gaussian": np.exp(-(X ** 2 + Y ** 2 + Z ** 2) / (2 * 0.05 ** 2)), "tail": np.exp(-9 * X - 6 * Y - 3 * Z) * (1 + 0.1 * noise)}
    for s in (1e-1, 1e-3, 1e-12):
        f[f"vertex {s:g}"] = np.where(vertex, 1.0, s * noise)
    for name, at in (("edge", edge), ("face", face), ("inner plane", inner)):
        for s in (0.2, 1e-3, 1e-9):
            f[f"{name} {s:g}"] = np.where(at, 1.0, s * noise)
    return f


def _product(G, B, u):
    """Exact product (long double) and the sums of the absolute values of its terms, (n_elt, n, n, n)."""
    L = np.longdouble

    def contract(G, B, u):
        g = [np.einsum("al,eajk->eljk", G, u), np.einsum("am,eiak->eimk", G, u), np.einsum("ap,eija->eijp", G, u)]
        idx = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
        v = [sum(B[..., idx[a][b]] * g[b] for b in range(3)) for a in range(3)]
        return (np.einsum("ia,eajk->eijk", G, v[0]) + np.einsum("ja,eiak->eijk", G, v[1])
                + np.einsum("ka,eija->eijk", G, v[2]))

    return (contract(G.astype(L), B.astype(L), u.astype(L)),
            contract(np.abs(G).astype(L), np.abs(B).astype(L), np.abs(u).astype(L)).astype(float))


class _Elements:
    """An operator of elements without common dofs, each with its factors and its field."""

    def __init__(self, order, seed=0):
        rng = np.random.default_rng([order, seed])
        n, self.order = order + 1, order
        fac, fld = _factors(order, rng), _fields(order, rng)
        self.names = [(a, b) for a in fac for b in fld]
        self.B = np.stack([fac[a] for a, _ in self.names])
        self.u = np.stack([fld[b] for _, b in self.names])
        self.G = _matrix(order)
        self.local = local_numbering(order).reshape(-1)  # [(i n + j) n + k] -> local index
        ne, Q = len(self.names), n ** 3
        nodle = np.arange(ne * Q, dtype=np.int32).reshape(ne, Q)
        b = np.zeros((ne, Q, 6))
        b[:, self.local] = self.B.reshape(ne, Q, 6)
        self.op = FemMatrixFreeOperator(order, nodle, b, ne * Q, "fp64", gradphi=self.G)

    def apply(self, u):
        ne = u.shape[0]
        x, y = np.zeros((ne, self.local.size)), np.zeros(u.size)
        x[:, self.local] = u.reshape(ne, -1)
        self.op.MltVector(x.reshape(-1), y)
        return y.reshape(ne, -1)[:, self.local].reshape(u.shape)


def _check(order, e, y, pipe):
    exact, absolute = _product(e.G, e.B, e.u)
    err, err_pipe = (y - exact).astype(float), (pipe - exact).astype(float)
    # one direction of the product is two contractions of n terms and a factor row in FP64: 2 (n + 1) + 4 roundings
    entry = (2 * (order + 2) + 4) * U * absolute
    norm = lambda a: np.sqrt((np.asarray(a, dtype=float) ** 2).sum(axis=(1, 2, 3)))
    for q, name in enumerate(e.names):
        assert (np.abs(err[q]) <= entry[q]).all(), (name, np.nanmax(np.abs(err[q]) / entry[q]))
    # both arithmetics round at random: twice the other's error, never below a last rounding of the result
    worst = norm(err) / np.maximum(np.maximum(norm(err_pipe), U * norm(exact)), 1e-300)
    bad = [(e.names[q], float(worst[q])) for q in np.nonzero(worst > 2.0)[0]]
    assert not bad, bad


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("seed", [0, 1])
def test_products_are_as_close_as_fp64(order, seed):
    e = _Elements(order, seed)
    assert e.op.tuning()["layout"] == "fixed_point"
    y = e.apply(e.u)
    e.op.set_variant(FP64_PIPE_TILE[order], 0)
    _check(order, e, y, e.apply(e.u))
    e.op.close()


@pytest.mark.parametrize("order", [1, 2, 4, 6, 8])
def test_an_element_does_not_see_the_others_of_its_tile(order):
    e = _Elements(order)
    y = e.apply(e.u)
    other = np.array([q % 2 == 1 for q in range(len(e.names))])
    u = e.u.copy()
    u[other] = np.roll(e.u, 3, axis=0)[other]
    u[1, 0, 0, 0] = np.inf
    assert np.array_equal(e.apply(u)[~other], y[~other])
    e.op.close()

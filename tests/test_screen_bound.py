"""The lower bound of K2 by which the genotype-split search leaves out triplets (epik2_test_screen_bound,
the search's FP32 arithmetic on the host).  It must never exceed the score, whatever the table and the
class split, and it must stay close enough to leave out most triplets also where alleles are rare or the
classes uneven: a triplet whose bound reaches the best score costs several times a screened one."""
import ctypes

import numpy as np
import pytest

import epik2
import oracle as O


def bounds(n0, n1, tables):
    t = np.ascontiguousarray(tables.reshape(len(tables), 54), dtype=np.uint32)
    out = np.empty(len(t), dtype=np.float32)
    assert epik2.library().epik2_test_screen_bound(n0, n1, t.ctypes.data_as(ctypes.c_void_p), len(t),
                                                   out.ctypes.data_as(ctypes.c_void_p)) == epik2.OK
    return out


def fp32_scores(tables):
    """K2 in the search's FP32 order: sum over the cells of (T[a+b+1] - T[a]) - T[b]."""
    lut = epik2.k2_lut(int(tables.sum(axis=(1, 2)).max()) + 2)
    a, b = tables[:, 0], tables[:, 1]
    terms = (lut[a + b + 1] - lut[a]) - lut[b]
    s = np.zeros(len(tables), np.float32)
    for c in range(27):
        s = (s + terms[:, c]).astype(np.float32)
    return np.abs(s)


def random_tables(rng, n0, n1, n):
    """Tables of given class sizes: from all samples in one cell to even ones, classes alike or apart."""
    out = np.zeros((n, 2, 27), np.int64)
    for t in range(n):
        w = rng.dirichlet(np.full(27, 10.0 ** rng.uniform(-2.5, 1)))
        tilt = rng.choice([0.0, 0.3, 3.0])
        v = w * np.exp(tilt * rng.standard_normal(27))
        out[t, 0] = rng.multinomial(n0, w)
        out[t, 1] = rng.multinomial(n1, v / v.sum())
    return out


SPLITS = [(1, 0), (0, 1), (1, 1), (3, 2), (40, 1), (100, 100), (700, 300), (30, 970), (3800, 200), (4000, 20),
          (1367, 2633), (8192, 8192), (65535, 65535), (65535, 30), (0, 65535), (20000, 65535)]


@pytest.mark.parametrize("n0,n1", SPLITS)
def test_never_above_the_score(n0, n1):
    rng = np.random.default_rng(n0 + 3 * n1)
    t = random_tables(rng, n0, n1, 400)
    one = np.zeros((54, 2, 27), np.int64)  # everyone in one cell; the classes in different cells
    for c in range(27):
        one[c, 0, c], one[c, 1, c] = n0, n1
        one[27 + c, 0, c], one[27 + c, 1, (c + 5) % 27] = n0, n1
    t = np.concatenate([t, one])
    b, s = bounds(n0, n1, t), fp32_scores(t)
    assert np.all(b <= s), (b - s).max()
    s64 = np.array([O.k2_fp64(x.reshape(54).astype(np.uint32)) for x in t])
    assert np.all(b <= s64), (b - s64).max()


@pytest.mark.parametrize("S,maf,cases", [(4000, (0.02, 0.05), 0.05), (4000, (0.005, 0.02), 0.05), (4000, (0.05, 0.5), 0.02),
                                         (1000, (0.02, 0.05), 0.05), (1000, (0.001, 0.005), 0.5),
                                         (4000, (0.0005, 0.002), 0.5), (16384, (0.05, 0.5), 0.05), (8192, (0.05, 0.5), 0.0061)])
def test_leaves_out_most_tables_of_rare_alleles_and_uneven_classes(S, maf, cases):
    """Of 3000 random triplets without an effect the bound of at most a quarter reaches the lowest score
    among them."""
    rng = np.random.default_rng(S + int(1000 * cases))
    M, n1 = 60, int(S * cases)
    p = rng.uniform(*maf, M)
    u = rng.random((S, M))
    g = (u >= (1 - p) ** 2).astype(int) + (u >= 1 - p * p)
    ph = np.zeros(S, bool)
    ph[rng.permutation(S)[:n1]] = True
    t = np.empty((3000, 2, 27), np.int64)
    for x in range(len(t)):
        i, j, k = rng.choice(M, 3, replace=False)
        cell = 9 * g[:, i] + 3 * g[:, j] + g[:, k]
        t[x] = np.bincount(cell[~ph], minlength=27), np.bincount(cell[ph], minlength=27)
    s = fp32_scores(t)
    reach = np.mean(bounds(S - n1, n1, t) <= s.min())
    assert reach <= 0.25, reach

"""The projector kernels along lines of cubes, the local pencils and the atom-matrix chain at the
edges of their ranges, against the oracle's FP64 action: every basis size and mixtures of them, block
lists longer than a work item, x-lines that are no multiple of a segment, sources without blocks near
an image, more images at a segment than its record stage holds, vectors off the 16-byte boundary and
z-lines beyond the pencils' limit.

Tolerances (largest error over the largest value): a value is a sum of at most a few thousand
products, so 1e-12 is some 5,000 FP64 roundings; FP32 3e-5 is some 500."""
import numpy as np
import pytest

import oracle
from helpers import geometry, inputs_for, product_plan, rel_err
from angstromcube_b200 import _lib, green_action

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 3e-5}


def with_numax(g, numax):
    for a, l in zip(g.xyzZinso, numax):
        a[5] = l
    return g


GEOMETRIES = {
    **{"numax%d" % l: (lambda l=l: geometry((4, 4, 4), (1, 1, 1), 6.0, (1, 1, 1), 4, 2, numax=l)) for l in (0, 1, 2, 4, 6, 7)},
    "mixed_to_5": lambda: with_numax(geometry((5, 4, 6), (1, 0, 2), 2.2, (2, 1, 1), 4, 6), (0, 5, 2, 3, 1, 4)),
    "mixed_to_7": lambda: with_numax(geometry((5, 4, 6), (1, 3, 0), 2.2, (1, 2, 1), 4, 4), (7, 0, 5, 6)),
    # one sphere over some 200 cubes, x-lines of up to 9 cubes, the source box in a corner of it
    "wide": lambda: geometry((11, 9, 10), (0, 0, 0), 3.6, (3, 1, 2), 4, 2, sigma=0.65, numax=5),
    # spheres that miss most sources' regions
    "apart": lambda: geometry((14, 3, 3), (2, 0, 0), 1.3, (14, 1, 1), 4, 3, sigma=0.4, numax=2),
    # every cube near dozens of images
    "crowded": lambda: geometry((3, 3, 3), (1, 1, 1), 6.0, (1, 1, 1), 4, 12, sigma=0.6, numax=2),
}


def plan_and_inputs(g, seed=3):
    Vc, mats, offs, E, k, dVol, _ = inputs_for(g)
    p = product_plan(g, Vc, mats, offs, E, k, dVol)
    x = np.random.default_rng(seed).standard_normal((p.nnzb, 2, 64, 64))
    return p, x, oracle.RestatedOracle(p.export(), Vc, E).action(x)


def apply(p, x_np, dtype, offset=0, columns=None):
    t = getattr(torch, dtype)
    n = x_np.size
    buf = [torch.zeros(n + offset, dtype=t, device="cuda") for _ in range(2)]
    x, y = (b[offset:].view(x_np.shape) for b in buf)
    x.copy_(torch.from_numpy(x_np))
    columns = p.export()["colindx"] if columns is None else columns
    ci = torch.from_numpy(columns.astype(np.int16)).cuda()
    green_action.action_t(p, dtype).multiply(y, x, ci, p.nnzb, p.nCols)
    torch.cuda.synchronize()
    return y.double().cpu().numpy()


@pytest.mark.parametrize("dtype", sorted(TOL))
@pytest.mark.parametrize("name", sorted(GEOMETRIES))
def test_action_at_the_edges(name, dtype):
    p, x, ref = plan_and_inputs(GEOMETRIES[name]())
    assert rel_err(apply(p, x, dtype), ref) < TOL[dtype]
    assert np.array_equal(apply(p, x, dtype), apply(p, x, dtype))      # sums in a fixed order


@pytest.mark.parametrize("chunk", [1, 2, 39, 40, 41])
@pytest.mark.parametrize("name", ["wide", "mixed_to_7"])
def test_work_items_of_every_length(name, chunk, monkeypatch):
    """Projection items of one position, of the most that fit an item's tables (40; 41 is cut to it) and
    lists that they divide unevenly."""
    monkeypatch.setenv("A43G_PRJ_CHUNK", str(chunk))
    p, x, ref = plan_and_inputs(GEOMETRIES[name]())
    lengths = np.diff(p.export()["SHOprj_start"].reshape(p.nCols, -1), axis=1)
    assert lengths.max() > 41 and (lengths % min(chunk, 40) != 0).any() == (chunk > 1)
    for dtype in TOL:
        assert rel_err(apply(p, x, dtype), ref) < TOL[dtype]
        assert np.array_equal(apply(p, x, dtype), apply(p, x, dtype))


@pytest.mark.parametrize("dtype", sorted(TOL))
def test_vectors_off_the_16_byte_boundary(dtype):
    """One element further, x and y take the projector kernels without 16-byte copies."""
    p, x, ref = plan_and_inputs(GEOMETRIES["mixed_to_5"]())
    assert rel_err(apply(p, x, dtype, offset=1), ref) < TOL[dtype]


@pytest.mark.parametrize("dtype,xo,yo", [("float64", 1, 0), ("float64", 0, 1), ("float64", 1, 1), ("float32", 2, 0),
                                         ("float32", 0, 2), ("float32", 1, 0), ("float32", 0, 1), ("float32", 3, 2)])
@pytest.mark.parametrize("name", ["mixed_to_5", "numax1"])
def test_pencils_off_the_16_byte_boundary(name, dtype, xo, yo):
    """The local part of x and y on any element is the pencils': the same sums in the same order as
    on 16 bytes (the rows kernel adds in another order).  A cell with a boundary of every kind and
    phases, and one whose lines of cubes are their own neighbours."""
    p, x_np, _ = plan_and_inputs(GEOMETRIES[name]())
    t = getattr(torch, dtype)
    y = []
    for a, b in ((0, 0), (xo, yo)):
        xs, ys = (torch.full((x_np.size + o + 4,), 7.0, dtype=t, device="cuda") for o in (a, b))
        xs[a:a + x_np.size] = torch.from_numpy(x_np.ravel()).to(t)
        _lib.check(_lib.lib().a43g_action_part(p.handle, 0, ys[b:].data_ptr(), xs[a:].data_ptr(), None,
                                               green_action.action_t(p, dtype).dtype), "local part")
        torch.cuda.synchronize()
        y.append(ys[b:b + x_np.size])
        assert (ys[:b] == 7).all() and (ys[b + x_np.size:] == 7).all()
    assert torch.equal(y[0], y[1])


@pytest.mark.parametrize("dtype", sorted(TOL))
@pytest.mark.parametrize("nz", [128, 129])
def test_longest_lines(nz, dtype):
    """The pencils hold 128 cubes of a z-line; longer ones take the rows kernel."""
    p, x, ref = plan_and_inputs(geometry((2, 1, nz), (1, 1, 1), 80.0, (1, 1, 1), 4, 0))
    assert p.nnzb == 2 * nz
    assert rel_err(apply(p, x, dtype), ref) < TOL[dtype]


@pytest.mark.parametrize("dtype", sorted(TOL))
@pytest.mark.parametrize("name", ["wide", "mixed_to_5", "mixed_to_7"])
def test_addition_reads_the_callers_columns(name, dtype):
    """The addition takes the coefficients of the columns that the caller names: here any source for
    any block, so that the cubes of a segment take different ones."""
    g = GEOMETRIES[name]()
    Vc, mats, offs, E, k, dVol, _ = inputs_for(g)
    p = product_plan(g, Vc, mats, offs, E, k, dVol)
    rng = np.random.default_rng(8)
    x = rng.standard_normal((p.nnzb, 2, 64, 64))
    e = p.export()
    e["colindx"] = rng.integers(0, p.nCols, p.nnzb).astype(e["colindx"].dtype)
    ref = oracle.RestatedOracle(e, Vc, E).action(x)
    assert rel_err(ref, oracle.RestatedOracle(p.export(), Vc, E).action(x)) > 1e-3
    assert rel_err(apply(p, x, dtype, columns=e["colindx"]), ref) < TOL[dtype]

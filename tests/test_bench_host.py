"""Host logic of bench.py that needs no GPU: the DRAM traffic table under profiles/ and the
naming of the local kernel the autotuner chose."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def load_bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_traffic_table_names_kernels_that_exist():
    """Every row is a kernel of the sources with its precision, moves at least its vectors (read once,
    written once) and is the committed capture's figure of the 4,096 blocks."""
    b = load_bench()
    with open(os.path.join(ROOT, "angstromcube_b200", "csrc", "action.cu")) as f:
        source = f.read()
    with open(os.path.join(ROOT, "profiles", "ncu_action_one_source.md")) as f:
        rows = [[c.strip(" `") for c in line.split("|")[1:-1]] for line in f if line.startswith("| ")]
    head, traffic = rows[0], next(r for r in rows if r[0].startswith("DRAM traffic"))
    keys = [k for k in ("local_pencil_kernel_f32", "local_pencil_kernel_f64") if b.read_traffic(k) is not None]
    with open(os.path.join(ROOT, "profiles", "traffic.txt")) as f:
        assert keys == [line.split()[0] for line in f if line.strip() and not line.startswith("#")]
    for key in keys:
        name, precision = key[:-4], key[-3:]
        assert name + "(" in source
        per_block = b.read_traffic(key)
        assert per_block >= 2 * 8192 * int(precision[1:]) / 8
        captured = float(traffic[head.index("local_pencil " + precision.upper().replace("F", "FP"))]) * 1e6 / 4096
        assert abs(per_block - captured) < 100            # the table gives 0.1 MB
    assert b.read_traffic("no_such_kernel") is None


def test_local_kernel_named_from_the_autotuner_choice():
    b = load_bench()
    line = "chosen: projector chunk 40, local %s, CUDA-core projector"
    name, key = b.local_kernel_of([line % "pencils"])
    assert name.startswith("local_pencil_kernel<float>") and key == "local_pencil_kernel_f32"
    name, key = b.local_kernel_of([line % "plain rows"])
    assert name.startswith("local_fused_kernel") and key is None
    with open(os.path.join(ROOT, "angstromcube_b200", "csrc", "autotune.cu")) as f:
        source = f.read()                                 # the line is the autotuner's
    assert 'chosen: projector chunk %u, local %s, %s projector' in source
    assert '"plain rows" : "pencils"' in source


def test_pair_walk_is_a_permutation_spread_over_the_contour():
    b = load_bench()
    order = b.pair_order(128)
    assert sorted(order) == list(range(128))
    # consecutive solves are far apart on the contour (energies are the outer loop, 4 k-points)
    assert all(abs(order[i + 1] // 4 - order[i] // 4) >= 8 for i in range(20))


def test_contour_workload():
    """32 Gauss-Legendre energies on the semicircle from -1 to 0 Ha (imaginary parts 2.1e-3 to
    0.5 Ha), 4 k-points, truncation radii clamp(8/sqrt(Im E/0.5), 8, 16); the weights integrate
    a constant and a linear function of E along the semicircle exactly."""
    import numpy as np
    from angstromcube_b200 import workloads
    w, pairs = workloads.batched_contour()
    assert len(pairs) == 128 and w.geometry.sources == (2, 2, 2)
    E = np.array([p[0] for p in pairs[::4]])
    assert 2e-3 < E.imag.min() < 2.2e-3 and 0.498 < E.imag.max() <= 0.5
    Es, ws = workloads.contour_semicircle(32)
    assert abs(ws.sum() - (0.0 - (-1.0))) < 1e-13          # integral of dE from -1 to 0
    assert abs((ws * Es).sum() - (0.0 - 1.0) / 2) < 1e-13  # integral of E dE
    rs = [p[3] for p in pairs]
    assert min(rs) > 8.0 and max(rs) == 16.0
    K, wk = workloads.contour_kpoints()
    assert np.all(K[0] == 0) and np.all(K[1:] < 0.5) and np.all(K[1:, 0] >= K[1:, 1]) and abs(wk.sum() - 1) < 1e-15

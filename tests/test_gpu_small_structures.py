"""Dispatch of structures that do not fill the GPU (split receivers, few-row GEMMs, shared components, one-call evaluation)
against the numpy oracle, at the sizes where its branches change."""
import numpy as np
import pytest
import torch

from oracle.mace_numpy import MaceOracle
from oracle.mace_numpy_deep import DeepMaceOracle
from symmetrix_b200 import MACE, _lib, structures as st
from symmetrix_b200.mace import SymmetrixError

pytestmark = pytest.mark.gpu

REL = {"float64": 1e-10, "float32": 1e-4}


def rel_err(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def expected(oracle, s, spec, numbers):
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, numbers)
    e, nf = oracle.compute_node_energies_forces(inputs)
    f, v = st.atom_forces_and_virial(inputs, nl, nf)
    return inputs, nl, np.asarray(e), f, v


def check(got, want, dtype):
    f, v, energy, e = got
    _, _, e_ref, f_ref, v_ref = want
    assert abs(energy - e_ref.sum()) <= REL[dtype] * abs(e_ref.sum())
    assert rel_err(e, e_ref) <= 10 * REL[dtype]
    assert rel_err(f, f_ref) <= 10 * REL[dtype]
    assert rel_err(v, v_ref) <= 100 * REL[dtype]


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("name,channels,cells", [
    ("fcc128", 128, [(1, 1, 1), (1, 1, 2), (1, 2, 2), (2, 3, 3), (3, 3, 5)]),     # 4 ... 180 atoms: 8, 8, 8, 4 and 1 CTAs per receiver
    ("fcc128", 33, [(1, 1, 2), (2, 2, 3)]),                                       # odd: the last pair of float channels is half empty
    ("large256", 65, [(1, 1, 2)]),                                                # the same with the adjoint in tensor memory
    ("fcc128", 40, [(1, 1, 2), (2, 2, 3)]),                                       # a second, partly filled GEMM tile
    ("large256", 160, [(1, 1, 1), (2, 2, 2)]),                                    # two channel blocks, nine components
    ("deep256", 32, [(1, 1, 1), (2, 2, 3)]),                                      # three blocks: products merged with typed residuals
])
def test_one_call_evaluation_matches_the_oracle(model_file, dtype, name, channels, cells):
    path, model, spec = model_file(name, num_channels=channels, num_spline_points=32)
    oracle = (DeepMaceOracle if name == "deep256" else MaceOracle)(model)
    ev = MACE(path, dtype=dtype)
    for c in cells:
        s = st.fcc_box(c, 3.6, model["atomic_numbers"], seed=sum(c))
        want = expected(oracle, s, spec, model["atomic_numbers"])
        types = want[0]["node_types"]
        check(ev.evaluate(s.positions, types, s.cell, s.pbc), want, dtype)


def test_one_call_evaluation_grows_and_shrinks(model_file):
    """Edge arrays and rows keep the capacity of earlier structures: more edges, longer rows than ever, fewer again, an open
    and an empty structure, on one handle; the neighbour list left behind is the host's."""
    path, model, spec = model_file("fcc128", num_channels=8, num_spline_points=32)
    oracle = MaceOracle(model)
    ev = MACE(path, dtype="float64")
    z = model["atomic_numbers"]
    open_box = st.fcc_box((2, 2, 3), 3.6, z, seed=3)
    open_box.pbc = (True, False, False)
    boxes = [st.fcc_box(1, 3.6, z, seed=1), st.fcc_box((3, 4, 4), 3.6, z, seed=2), st.fcc_box(2, 2.5, z, jitter=0.05, seed=3),
                  st.fcc_box((1, 1, 2), 3.6, z, seed=4), open_box]
    for s in boxes:
        want = expected(oracle, s, spec, z)
        check(ev.evaluate(s.positions, want[0]["node_types"], s.cell, s.pbc), want, "float64")
        edges = ev.get_edges()
        np.testing.assert_array_equal(edges["neigh_indices"], want[1]["j"])
        np.testing.assert_array_equal(edges["shifts"], want[1]["S"])
        np.testing.assert_array_equal(edges["r"], want[1]["d"])
    f, v, energy, e = ev.evaluate(np.zeros((0, 3)), np.zeros(0, np.int32), np.eye(3) * 9.0)
    assert f.shape == (0, 3) and e.size == 0 and energy == 0.0 and not v.any()


@pytest.mark.parametrize("name", ["fcc128", "large256"])
def test_evaluators_of_different_widths_take_turns(model_file, name):
    """The split forward kernels ask for shared memory by the width of the model; a narrower evaluator in the same process must
    not lower what the wider one may ask for, whichever of them came first."""
    evs = {k: MACE(model_file(name, num_channels=k, num_spline_points=32)[0], dtype="float64") for k in (128, 32, 64)}
    s = st.fcc_box((1, 1, 2), 3.6, model_file(name, num_channels=32, num_spline_points=32)[1]["atomic_numbers"], seed=3)
    types = np.arange(s.num_atoms, dtype=np.int32) % 2
    first = {k: ev.evaluate(s.positions, types, s.cell, s.pbc)[0].copy() for k, ev in evs.items()}
    for k, ev in evs.items():
        np.testing.assert_array_equal(ev.evaluate(s.positions, types, s.cell, s.pbc)[0], first[k])


@pytest.mark.parametrize("cells_away", [600, -600, 5000])
def test_atoms_too_far_outside_the_cell_are_refused(model_file, cells_away):
    """A shift that the sort keys have no room for is reported before any edge is made of it, by the one-call evaluation (which
    learns of it with the results) and by the neighbour list, and the handle goes on."""
    path, model, _ = model_file("fcc128", num_channels=8, num_spline_points=32)
    ev = MACE(path, dtype="float64")
    s = st.fcc_box(2, 3.6, model["atomic_numbers"], seed=5)
    types = np.arange(s.num_atoms, dtype=np.int32) % 3
    before = ev.evaluate(s.positions, types, s.cell, s.pbc)
    far = s.positions.copy()
    far[3] += cells_away * s.cell[0]
    for call in (ev.evaluate, ev.build_neighbors, ev.evaluate):
        with pytest.raises(SymmetrixError) as err:
            call(far, types, s.cell, s.pbc)
        assert err.value.status == _lib.SMX_ERR_INVALID_ARGUMENT
    after = ev.evaluate(s.positions, types, s.cell, s.pbc)
    np.testing.assert_array_equal(after[0], before[0])
    assert after[2] == before[2]


def test_no_edge_set_is_left_by_a_call_that_failed_on_the_way(model_file):
    """A neighbour list that is refused after the old arrays were given up leaves no edge set: stages say so instead of running the
    new number of atoms over the old rows. A call whose arguments are refused leaves the old set as it was."""
    path, model, _ = model_file("fcc128", num_channels=8, num_spline_points=32)
    ev = MACE(path, dtype="float64")
    z = model["atomic_numbers"]
    small, large = st.fcc_box((1, 1, 2), 3.6, z, seed=6), st.fcc_box((2, 2, 3), 3.6, z, seed=7)
    types = [np.arange(s.num_atoms, dtype=np.int32) % 2 for s in (small, large)]
    ev.build_neighbors(small.positions, types[0], small.cell, small.pbc)
    with pytest.raises(SymmetrixError):
        ev.build_neighbors(large.positions, types[1], large.cell, large.pbc, r_cut=-1.0)
    ev.compute_current()                                    # refused before anything was replaced
    e = ev.node_energies
    far = large.positions.copy()
    far[0] += 600 * large.cell[1]
    for call in (ev.build_neighbors, ev.evaluate):
        ev.build_neighbors(small.positions, types[0], small.cell, small.pbc)
        with pytest.raises(SymmetrixError):
            call(far, types[1], large.cell, large.pbc)
        with pytest.raises(SymmetrixError) as err:
            ev.compute_current()
        assert err.value.status == _lib.SMX_ERR_INVALID_ARGUMENT and "no edge set" in str(err.value)
    ev.build_neighbors(small.positions, types[0], small.cell, small.pbc)
    ev.compute_current()
    np.testing.assert_array_equal(ev.node_energies, e)


def test_an_allocation_that_fails_is_reported_once(model_file):
    """512 GB of feature rows are refused by the allocator; the calls after it find no error of their own."""
    path, model, _ = model_file("fcc128", num_channels=8, num_spline_points=32)
    ev = MACE(path, dtype="float64")
    s = st.fcc_box((1, 1, 2), 3.6, model["atomic_numbers"], seed=6)
    types = np.zeros(s.num_atoms, dtype=np.int32)
    want = ev.evaluate(s.positions, types, s.cell, s.pbc)
    with pytest.raises(SymmetrixError) as err:
        ev.resize_rows("H1", 2_000_000_000)
    assert err.value.status == _lib.SMX_ERR_CUDA
    got = ev.evaluate(s.positions, types, s.cell, s.pbc)
    np.testing.assert_array_equal(got[0], want[0])


def test_memory_of_an_evaluation_follows_its_edges(model_file):
    """8,000 atoms with six neighbours each: the one-call evaluation takes the memory that the same edges take when they are given
    (64 edges per atom, taken for granted, would be another gigabyte of messages)."""
    path, model, spec = model_file("fcc128", num_channels=64, num_spline_points=32)
    g = np.arange(8000)
    pos = 4.0 * np.stack([g % 20, g // 20 % 20, g // 400], 1)
    s = st.Structure(pos, np.diag([80.0] * 3), np.full(8000, model["atomic_numbers"][0]), (True, True, True))
    types, rc = np.zeros(8000, np.int32), 4.9      # 16 bins an axis: the one-CTA index kernels

    def used():
        free, total = torch.cuda.mem_get_info()
        return total - free

    ev = MACE(path, dtype="float64")
    start = used()
    got = ev.evaluate(s.positions, types, s.cell, s.pbc, r_cut=rc)
    one_call = used() - start
    edges = ev.get_edges()
    assert edges["r"].size == 6 * 8000
    ev.close()
    ev = MACE(path, dtype="float64")
    start = used()
    ev.compute_node_energies_forces(8000, types, *[edges[k] for k in ("num_neigh", "neigh_indices", "neigh_types")], edges["xyz"].reshape(-1), edges["r"])
    forces, _, energy = ev.reduce_forces()
    given = used() - start
    assert one_call <= given + 2**28
    assert abs(got[2] - energy) <= 1e-12 * abs(energy)


@pytest.mark.parametrize("atoms,spacing", [(7000, 3.3), (40000, 6.0)])
def test_a_dense_cluster_in_a_large_sparse_box(model_file, atoms, spacing):
    """Rows far longer than the others, in more atoms than may all have rows of that length: they are found a second time at their
    own offsets, for a structure of the one-CTA index kernels and for a larger one. The list is the host's, bit for bit, and the
    memory is not that of all rows as long as the longest."""
    path, model, _ = model_file("fcc128", num_channels=8, num_spline_points=32)
    rng, cluster = np.random.default_rng(atoms), 600
    side = int(np.ceil(atoms ** (1 / 3)))
    g = np.arange(atoms - cluster)
    pos = spacing * np.stack([g % side, g // side % side, g // side ** 2], 1) + rng.normal(0, 0.3, (atoms - cluster, 3))
    pos = np.concatenate([pos, 0.5 * spacing * side + rng.uniform(-1.0, 1.0, (cluster, 3))])
    s = st.Structure(pos, np.diag([spacing * side] * 3), np.full(atoms, model["atomic_numbers"][0]), (True, True, True))
    types, rc = np.zeros(atoms, np.int32), 4.0
    nl = st.neighbor_list(s, rc)
    ev = MACE(path, dtype="float32")
    start = torch.cuda.mem_get_info()[0]
    got = ev.evaluate(s.positions, types, s.cell, s.pbc, r_cut=rc)
    taken = start - torch.cuda.mem_get_info()[0]
    edges = ev.get_edges()
    np.testing.assert_array_equal(edges["neigh_indices"], nl["j"])
    np.testing.assert_array_equal(edges["shifts"], nl["S"])
    np.testing.assert_array_equal(edges["r"], nl["d"])
    assert edges["num_neigh"].max() >= cluster - 1
    again = MACE(path, dtype="float32")
    start = torch.cuda.mem_get_info()[0]
    again.compute_node_energies_forces(atoms, types, *[edges[k] for k in ("num_neigh", "neigh_indices", "neigh_types")], edges["xyz"].reshape(-1), edges["r"])
    assert abs(got[2] - again.reduce_forces()[2]) <= 1e-6 * abs(got[2])
    assert taken <= start - torch.cuda.mem_get_info()[0] + 2**27          # 40,000 rows of 704 keys are 225 MB


@pytest.mark.parametrize("channels,cells", [(33, (5, 6, 10)), (160, (2, 4, 7)), (160, (2, 4, 8))])
def test_float_forward_pass_of_degree_two_changes_lanes(model_file, channels, cells):
    """L_max = 2, float32, on both sides of the line (37,888 channels of atoms on 148 SMs) where the forward tensor product goes from
    pairs of channels to single ones: 1,200 atoms of 33 channels, 224 and 256 of 160, which are two chunks. One neighbour shell."""
    path, model, spec = model_file("large256", num_channels=channels, num_spline_points=32)
    s = st.fcc_box(cells, 5.4, model["atomic_numbers"], seed=sum(cells))
    want = expected(MaceOracle(model), s, spec, model["atomic_numbers"])
    check(MACE(path, dtype="float32").evaluate(s.positions, want[0]["node_types"], s.cell, s.pbc), want, "float32")


def test_edges_without_their_opposite(model_file):
    """The two directions of a pair are tested with differently rounded distances, so a cutoff between the two keeps one edge of
    the pair alone. The senders' lists cannot be read off the receivers' rows then: both entries sort instead."""
    path, model, _ = model_file("fcc128", num_channels=8, num_spline_points=32)
    s = st.fcc_box(2, 3.6, model["atomic_numbers"], seed=21, jitter=0.2)
    nl = st.neighbor_list(s, 5.5)
    r2 = {(i, j, *S): (D[0] * D[0] + D[1] * D[1]) + D[2] * D[2] for i, j, S, D in zip(nl["i"], nl["j"], nl["S"].tolist(), nl["D"])}
    rc = 0.0
    for (i, j, a, b, c), x in r2.items():
        y = r2.get((j, i, -a, -b, -c), x)
        near = np.sqrt(y)
        for t in (near, np.nextafter(near, 0.0), np.nextafter(near, 9.0)):
            if 5.0 < t and x < t * t <= y:
                rc = float(t)
    nl = st.neighbor_list(s, rc)
    edges = {(i, j, *S) for i, j, S in zip(nl["i"], nl["j"], nl["S"].tolist())}
    assert any((j, i, -a, -b, -c) not in edges for i, j, a, b, c in edges)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    e, nf = MaceOracle(model).compute_node_energies_forces(inputs)
    f, v = st.atom_forces_and_virial(inputs, nl, nf)
    want = (inputs, nl, np.asarray(e), f, v)
    ev = MACE(path, dtype="float64")
    for _ in range(2):
        check(ev.evaluate(s.positions, inputs["node_types"], s.cell, s.pbc, r_cut=rc), want, "float64")
        np.testing.assert_array_equal(ev.get_edges()["neigh_indices"], nl["j"])
    ev.build_neighbors(s.positions, inputs["node_types"], s.cell, s.pbc, r_cut=rc)
    ev.compute_current()
    forces, virial, energy = ev.reduce_forces()
    check((forces, virial, energy, ev.node_energies), want, "float64")


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("base,copies", [((3, 3, 3), (1, 1, 11)), ((4, 4, 4), (2, 4, 4))])
def test_one_call_evaluation_of_thousands_of_atoms(model_file, dtype, base, copies):
    """From 1,185 atoms on (here 1,188) a row is one warp's, up to 8,192 (here all of them) one CTA builds the index arrays: copies of
    a cell give the cell's energies and forces."""
    path, model, spec = model_file("fcc128", num_channels=8, num_spline_points=32)
    cell = st.fcc_box(base, 5.4, model["atomic_numbers"], seed=22)
    _, _, e, f, v = expected(MaceOracle(model), cell, spec, model["atomic_numbers"])
    s, n = st.replicate(cell, copies), int(np.prod(copies))
    zmap = {z: t for t, z in enumerate(model["atomic_numbers"])}
    types = np.array([zmap[int(z)] for z in s.numbers], np.int32)
    want = (None, None, np.tile(e, n), np.tile(f, (n, 1)), n * v)
    check(MACE(path, dtype=dtype).evaluate(s.positions, types, s.cell, s.pbc), want, dtype)

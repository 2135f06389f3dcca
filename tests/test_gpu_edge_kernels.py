"""Edge kernels at the row widths where their lanes, groups and channel chunks end, against the oracle. All tests need a GPU."""
import numpy as np
import pytest
import torch

from oracle.mace_numpy import MaceOracle
from symmetrix_b200 import MACE, Symmetrix, structures as st
from tests.test_gpu_parity import INPUT_KEYS, _oracle_for, check_against, rel_err, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("L_max,channels", [
    (0, 1), (0, 31), (0, 64), (1, 5), (1, 33), (1, 62), (1, 64), (1, 65), (1, 129), (1, 130), (1, 258), (2, 7), (2, 34), (2, 130),
])
def test_row_widths(model_file, dtype, L_max, channels):
    """Odd rows of floats end in half a lane; 32, 64 and 128 lanes are where groups of warps and channel chunks begin."""
    path, model, spec = model_file("fcc128", num_channels=channels, num_spline_points=32, L_max=L_max)
    s = st.fcc_box(2, 3.6, model["atomic_numbers"], seed=channels)
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    e_ref, f_ref = _oracle_for(path, model)(inputs)
    e, f = run(MACE(path, dtype=dtype), inputs)
    check_against(dtype, e, f, e_ref, f_ref)


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("channels", [5, 66])
def test_row_widths_of_degree_three(model_file, dtype, channels):
    """Pairs of channels in the register kernel: odd rows add up over channels through shuffles, even ones through shared memory."""
    test_row_widths(model_file, dtype, 3, channels)


@pytest.mark.parametrize("spacing,jitter", [(5.4, 0.0), (3.2, 0.25), (2.5, 0.1), (2.0, 0.1), (1.7, 0.1)])
def test_zbl_rounds_of_a_receiver(model_file, spacing, jitter):
    """Rows with no pair inside the radii, with less than one round of 32, and with up to five (163 pairs)."""
    path, model, spec = model_file("fcc128", num_channels=32, num_spline_points=32, zbl=True)
    s = st.fcc_box(2, spacing, model["atomic_numbers"], seed=2, jitter=jitter)
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    o = MaceOracle(model)
    o._edges(inputs)
    o.node_energies, o.node_forces = np.zeros(o.N), np.zeros((o.r.size, 3))
    o.compute_ZBL()
    ev = MACE(path)
    ev.begin(*(inputs[k] for k in INPUT_KEYS))
    ev.compute_ZBL()
    # sums of up to 163 terms, each a polynomial in x^p that cancels to a part in a hundred and a few functions good to an ulp or two
    np.testing.assert_allclose(ev.node_energies, o.node_energies, rtol=1e-12, atol=1e-12 * np.abs(o.node_energies).max())
    np.testing.assert_allclose(ev.node_forces.reshape(-1, 3), o.node_forces, rtol=1e-12, atol=1e-12 * np.abs(o.node_forces).max())


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("name,channels,atoms", [
    ("organic128", 1, 9), ("organic128", 15, 9), ("organic128", 33, 9), ("organic128", 72, 9), ("organic128", 128, 18), ("organic128", 128, 144),
    ("organic128", 130, 27), ("organic128", 250, 9), ("organic128", 256, 36), ("organic128", 257, 9),
])
def test_last_block_in_one_launch(model_file, dtype, name, channels, atoms):
    """Whole evaluations of small structures run M1 to its adjoint in one launch, stages one launch each: both must give every array of
    the last block alike, at slices of the channels that end early or cover whole warps."""
    path, model, spec = model_file(name, num_channels=channels, num_spline_points=32)
    s = st.molecular_liquid(atoms // 9, seed=atoms)
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    one, each = MACE(path, dtype=dtype), MACE(path, dtype=dtype)
    each.set_profiling(True)           # times every stage, hence a launch for each
    e1, f1 = run(one, inputs)
    e2, f2 = run(each, inputs)
    assert one.launch_count < each.launch_count or channels > 256 or atoms * channels > 128 * 148
    # the same sums in another order: 128 products each in the precision of the evaluator, through two matrix products and a sigmoid
    rel = 1e-12 if dtype == "float64" else 2e-5
    assert rel_err(e1, e2) <= rel and rel_err(f1, f2) <= rel
    for field in ["M1", "H2", "H2_adj", "M1_adj", "A1_adj", "H1_adj"]:
        assert rel_err(getattr(one, field), getattr(each, field)) <= rel, field


def last_block_ctas(channels, atoms, dtype):
    """CTAs per node of the one launch that runs M1 to its adjoint, 0 where the stages are launches of their own: beyond four nodes per SM,
    128 SMs' worth of channels of nodes or 256 channels, and where a CTA would have a node of more than 160 channels to itself."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if atoms > 4 * sms or atoms * channels > 128 * sms or channels > 256:
        return 0
    room = sms * (1 if dtype == "float64" and channels > 128 else 2)
    c = 8
    while c > 1 and (atoms * c > room or channels < 16 * c):
        c //= 2
    return 0 if c == 1 and channels > 160 else c


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("channels,atoms", [
    (1, 9), (15, 9), (33, 9), (72, 9), (128, 18), (128, 144), (130, 27), (250, 9), (256, 36), (257, 9),
    (64, 153), (128, 153), (4, 585), (4, 603), (160, 81), (192, 81),
])
def test_lines_of_the_last_block_in_one_launch(model_file, dtype, channels, atoms):
    """The launches are merged up to the lines and not beyond, with a cluster per node or one CTA; where they are, every array of the last
    block is what matrix products give for copies of the structure beyond every line."""
    path, model, spec = model_file("organic128", num_channels=channels, num_spline_points=32)
    s = st.molecular_liquid(atoms // 9, seed=atoms)
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    one, each = MACE(path, dtype=dtype), MACE(path, dtype=dtype)
    each.set_profiling(True)           # times every stage, hence a launch for each
    e1, f1 = run(one, inputs)
    run(each, inputs)
    merged = last_block_ctas(channels, atoms, dtype) > 0
    assert each.launch_count - one.launch_count == (4 if merged else 0)
    if not merged:
        return
    # the same sums in another order: 128 products each in the precision of the evaluator, through two matrix products and a sigmoid
    rel = 1e-12 if dtype == "float64" else 2e-5
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    copies = 4 * sms // atoms + 1
    many = {k: np.tile(inputs[k], copies) for k in INPUT_KEYS if k != "num_nodes"}
    many["num_nodes"] = atoms * copies
    many["neigh_indices"] = many["neigh_indices"] + np.repeat(np.arange(copies) * atoms, inputs["neigh_indices"].size).astype(np.int32)
    large = MACE(path, dtype=dtype)
    e3, f3 = run(large, many)
    assert rel_err(e1, e3[:e1.size]) <= rel and rel_err(f1, f3[:f1.size]) <= rel
    for field in ["M1", "H2", "H2_adj", "M1_adj", "A1_adj", "H1_adj"]:
        got = getattr(one, field)
        assert rel_err(got, getattr(large, field)[:got.size]) <= rel, field


TWO_BLOCK_STAGES = ["compute_Y", "compute_R0", "compute_A0", "compute_M0", "compute_H1", "compute_R1", "compute_Phi1", "compute_A1", "compute_M1",
                    "compute_H2", "compute_readouts", "reverse_H2", "reverse_M1", "reverse_A1", "reverse_Phi1", "reverse_H1", "reverse_M0", "reverse_A0"]


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("channels,atoms", [(1, 9), (15, 9), (33, 9), (72, 9), (128, 9), (128, 144), (130, 27), (256, 36), (128, 207)])
def test_timed_stages_and_stage_calls_give_the_same_bits(model_file, dtype, channels, atoms):
    """A whole evaluation, one whose stages are timed and a sequence of stage calls: what is launched differs for small structures (all
    but the last case), the results do not. In float32 that holds up to where messages are added to the senders in any order."""
    path, model, spec = model_file("organic128", num_channels=channels, num_spline_points=32)
    s = st.molecular_liquid(atoms // 9, seed=atoms)
    nl = st.neighbor_list(s, spec.r_cut)
    inputs = st.evaluator_inputs(s, nl, model["atomic_numbers"])
    whole, timed, staged = (MACE(path, dtype=dtype) for _ in range(3))
    run(whole, inputs)
    timed.set_profiling(True)
    run(timed, inputs)
    staged.begin(*(inputs[k] for k in INPUT_KEYS))
    for stage in TWO_BLOCK_STAGES:
        kw = {"zero_H1_adj": False} if stage == "reverse_H2" else {"zero_dxyz": False, "zero_H1_adj": False} if stage == "reverse_Phi1" else {}
        getattr(staged, stage)(**kw)
    fields = ["node_energies", "A1", "M1", "H2", "H2_adj", "M1_adj", "A1_adj"]
    if dtype == "float64":
        fields += ["H1_adj", "M0_adj", "A0_adj", "node_forces"]
    assert set(timed.stage_times()) == {n for n in TWO_BLOCK_STAGES if n not in ("compute_Y", "compute_R0", "compute_R1")}
    for field in fields:
        want = getattr(whole, field)
        assert np.array_equal(getattr(timed, field), want), field
        assert np.array_equal(getattr(staged, field), want), field


@pytest.mark.parametrize("L_max,channels,cells", [(1, 66, (7, 7, 6)), (1, 67, (7, 7, 6)), (2, 130, (5, 5, 6))])
def test_contraction_on_pairs_of_channels(model_file, L_max, channels, cells):
    """float32 structures large enough for the contraction on pairs (of which the odd row has none), with node groups that end inside
    a type: against float64, whose contraction is another instantiation. Bounds as for the other float32 comparisons."""
    path, model, spec = model_file("fcc128", num_channels=channels, num_spline_points=32, L_max=L_max)
    s = st.fcc_box(cells, 3.6, model["atomic_numbers"], seed=3)
    assert s.num_atoms * channels > 4 * 128 * 148
    res = {}
    for dtype in ("float64", "float32"):
        calc = Symmetrix(path, dtype=dtype)
        calc.calculate(s.positions, s.cell, s.numbers, s.pbc)
        res[dtype] = (calc.results["forces"], calc.evaluator.M0, calc.evaluator.A0_adj)
    for got, want in zip(res["float32"], res["float64"]):
        assert rel_err(got, want) <= 1e-4


@pytest.mark.parametrize("cells", [(6, 6, 6), (5, 5, 10)])
def test_reverse_contraction_of_nine_components(model_file, cells):
    """float32: pairs of channels from 8/5 CTAs of them per SM on, between the two sizes; single channels below. Against float64, as above."""
    path, model, spec = model_file("fcc128", num_channels=66, num_spline_points=32, L_max=2)
    s = st.fcc_box(cells, 3.6, model["atomic_numbers"], seed=3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert s.num_atoms * 66 > 2 * 128 * sms
    assert (5 * (s.num_atoms + 5) * 33 <= 8 * 128 * sms) == (cells == (6, 6, 6))       # five element types
    res = {}
    for dtype in ("float64", "float32"):
        calc = Symmetrix(path, dtype=dtype)
        calc.calculate(s.positions, s.cell, s.numbers, s.pbc)
        res[dtype] = (calc.results["forces"], calc.evaluator.M0, calc.evaluator.A0_adj)
    for got, want in zip(res["float32"], res["float64"]):
        assert rel_err(got, want) <= 1e-4


@pytest.mark.parametrize("L_max,channels", [(0, 2), (0, 31), (0, 32), (0, 34), (0, 96), (0, 97), (0, 98),
                                             (1, 2), (1, 15), (1, 32), (1, 34), (1, 63), (1, 65)])
@pytest.mark.parametrize("cells", [(3, 3, 3), (6, 6, 6), (10, 10, 10)])
def test_reverse_of_narrow_rows(model_file, L_max, channels, cells):
    """float32: narrow even rows run on single channels in large structures and on pairs in small ones, with lines at 480 and 2,500 edges per
    SM (16 more per receiver) and at 32 and 96 channels; narrow odd rows change the way of their sums over channels at the first line.
    Against float64, which has one form. Bounds as for the other float32 comparisons."""
    path, model, spec = model_file("fcc128", num_channels=channels, num_spline_points=32, L_max=L_max)
    s = st.fcc_box(cells, 3.6, model["atomic_numbers"], seed=4)
    res = {}
    for dtype in ("float64", "float32"):
        calc = Symmetrix(path, dtype=dtype)
        calc.calculate(s.positions, s.cell, s.numbers, s.pbc)
        res[dtype] = (calc.results["forces"], calc.evaluator.H1_adj, calc.evaluator.node_forces)
    load = 78 * s.num_atoms + 16 * s.num_atoms
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sides = {(3, 3, 3): (0, 480), (6, 6, 6): (480, 2500), (10, 10, 10): (2500, 1 << 30)}[cells]
    assert sides[0] * sms <= load < sides[1] * sms
    for got, want in zip(res["float32"], res["float64"]):
        assert rel_err(got, want) <= 1e-4

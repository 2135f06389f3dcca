"""Edge kernels at the row widths where their lanes, groups and channel chunks end, against the oracle. All tests need a GPU."""
import pytest

from symmetrix_b200 import MACE, structures as st
from tests.test_gpu_parity import _oracle_for, check_against, run

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

"""LU-SGS version 5 marks an edge word that is not stored yet by a NaN.  A state's NaN must not be taken
for a missing term, neither that of all ones (memory filled with 0xFF), whose payload arithmetic
carries on, nor the signalling NaN of the mark itself: the step ends with the NaN report and its cell,
not with a timed-out wait, and the other solves of the handle are unharmed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WORDS = [-1, 0x7ff25ec0de5c0ffe]  # all ones; the mark (LU5_EMPTY)


def poison(s, word):
    """The word in every variable of one cell of a tile's last column (8 x 4 columns; 4 ghost layers)."""
    u = s.get_state(0)
    u.view(np.int64)[4 + 3, 4 + 7, 4 + 5] = word
    s.set_state(0, u)


@pytest.mark.parametrize("word", WORDS)
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("turb", [-1, 2, 3])
def test_the_nan_is_reported_as_a_nan(gpu, turb, prec, word):
    from meshes import wavy_box
    from test_gpu_lu_v5 import make
    p, _ = make(turb, prec, (4, 4, 4))
    case = wavy_box(12, 20, 11)  # 3 x 3 tiles
    s = gpu.Solver(p, case)
    assert s.lu_kernel_version() == 5
    poison(s, word)
    s.compute_residual(True)
    with pytest.raises(FloatingPointError) as e:
        s.residual()
    assert "block 1" in str(e.value)
    if turb < 0:  # good input again: the edge words are all empty, the bits are a new handle's (no mu kept from before)
        ref = gpu.Solver(p, case)
        s.init_flow()
        for h in (s, ref):
            h.compute_residual(True)
        assert np.array_equal(s.get_array(0, "DU")[0], ref.get_array(0, "DU")[0])
        ref.close()
    s.close()


@pytest.mark.parametrize("word", WORDS)
def test_the_other_solves_of_a_batch_go_on(gpu, word):
    from meshes import wavy_box
    from test_gpu_lu_v5 import make
    p, _ = make(0, 0, (4, 4, 4))
    case = wavy_box(12, 20, 11)
    s, ref = gpu.Batch([(p, case), (p, case)]), gpu.Batch([(p, case), (p, case)])
    poison(s, word)
    for h in (s, ref):
        h.advance(2)
    rms = s.residual_all()[1]  # raises on a timed-out wait
    assert np.isnan(rms[0]).any() and np.isfinite(rms[1]).all()
    assert np.array_equal(s.get_state(1), ref.get_state(1))
    s.close()
    ref.close()

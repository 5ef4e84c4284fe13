"""The cell lists of the beam grid: each cell's beams in strictly descending order (the order of the
reference's lists, which the reductions' shuffles start from), whatever the number of entries and cells."""
import numpy as np
import pytest

from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


@pytest.mark.gpu
@pytest.mark.parametrize("light_paths,res", [(3, 1), (3, 64), (5000, 2), (5000, 100)])
def test_cell_lists_descend(light_paths, res):
    w = W.generate(W.cube_scene("order", 8, 8, light_paths, 6, 0.02, techniques=W.BPT | W.BB1D), 0)
    with engine.EstimatorStage(0, engine.MODE_PLAIN) as st:
        st.set_bb1d_grid(res)
        st.run(w)
        g = st.grid_structure()
    cells, beams = g["cells"].astype(np.int64), g["beams"].astype(np.int64)
    assert cells[0] == 0 and cells[-1] == len(beams) and (np.diff(cells) >= 0).all()
    cell = np.repeat(np.arange(len(cells) - 1), np.diff(cells))
    same = cell[1:] == cell[:-1]
    assert same.any() and (np.diff(beams)[same] < 0).all()
    # every beam lies in the grid's box, so in at least one cell
    assert (np.unique(beams) == np.arange(len(w["beam_length"]))).all()

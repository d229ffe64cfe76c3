"""The simulation-information file (_info.txt) in the reference's format.

tests/golden/info_golden.json holds texts that the reference's own reader
(post/fileTreat.py getSimInfo, src/saveData.cu:469-613 writes the format) was
checked to parse into the descriptions' values when the fixture was made
(tests/golden/make_info_golden.py).  The library must still write exactly
these texts (mrlbm_info_text, the text mrlbm_save_info writes but for the step
geometry, which is the domain's own there); when the
environment variable MRLBM_REFERENCE names a reference checkout, the
reference's reader parses them again here.
"""
import json
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
import make_info_golden as mig  # noqa: E402


def golden():
    with open(os.path.join(HERE, "golden", "info_golden.json")) as f:
        return json.load(f)


def test_info_text_is_the_golden_text():
    g = golden()
    for key, d, sim_id, case_name, nsteps, mlups in mig.cases():
        assert mig.mrlbm.info_text(d, sim_id, case_name, nsteps, mlups) == g[key]["text"], key


def test_reference_reader_parses_the_info_text(tmp_path):
    ref = os.environ.get("MRLBM_REFERENCE")
    if not ref or not os.path.exists(os.path.join(ref, "post", "fileTreat.py")):
        pytest.skip("MRLBM_REFERENCE does not name a reference checkout")
    ft = mig.reference_parser(ref)
    g = golden()
    for key, d, sim_id, case_name, nsteps, mlups in mig.cases():
        text = mig.mrlbm.info_text(d, sim_id, case_name, nsteps, mlups)
        assert mig.parse_with_reference(ft, text, str(tmp_path / key), sim_id) == g[key]["parsed"], key


@pytest.mark.gpu
@pytest.mark.parametrize("shape,lattice", [((64, 64, 64), 19), ((128, 128, 128), 27), ((160, 160, 160), 19)])
def test_the_saved_text_has_the_chunk_that_runs(tmp_path, shape, lattice):
    """The plain march, the sums march and the three-CTA shape: BZ is the z
    chunk that the domain is stepped with, chosen or set."""
    m = mig.mrlbm
    dom = m.Domain(m.make_desc(*shape, lattice=lattice, tau=0.8))
    for chunk in (0, 7):
        dom.set_z_chunk(chunk)
        dom.save_info(str(tmp_path), "007", "runtime", 10, 1.0)
        text = (tmp_path / "007" / "007_info.txt").read_text()
        bz = [line.split(":")[1].strip() for line in text.splitlines() if line.strip().startswith("BZ:")]
        assert bz == [str(dom.z_chunk())], (bz, dom.z_chunk())
        assert not chunk or dom.z_chunk() == chunk
    dom.close()

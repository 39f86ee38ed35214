"""The plan of the lane-per-group fill on CPU: items, storage, waits and D
writes as lcg_host::prep_pair lays them out, walked with every access checked
and compared with a group-by-group evaluation (tests/cpp/lane_plan_demo.cu)."""
import os
import subprocess

import pytest

from locarna_gb300.synth import make_homolog, make_rna

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lane_demo():
    from locarna_gb300.build import GENCODE, NVCC, OUT, _run, build_engine
    build_engine()
    exe = os.path.join(OUT, "lane_plan_demo")
    _run([NVCC, GENCODE, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "cpp", "lane_plan_demo.cu"), "-o", exe,
          "-L", OUT, "-llocarna_gb300", "-Xlinker", "-rpath=" + OUT])
    return exe


# lengths around the column blocks (8) and row quads (4), uneven pairs, wide
# and narrow bands, gap openings down to none, and the modes that change which
# D entries a group writes
@pytest.mark.parametrize("groups", [32, 64])
@pytest.mark.parametrize("la,lb,homolog,nolp,stacking,max_diff,opening", [
    (16, 17, 0, 0, 0, -1, -750), (24, 31, 0, 0, 0, -1, -750), (40, 33, 0, 0, 0, -1, 0),
    (57, 60, 0, 0, 0, -1, -750), (64, 64, 1, 0, 1, -1, -750), (63, 65, 1, 1, 0, -1, -750),
    (72, 80, 1, 1, 1, -1, -750), (100, 41, 0, 0, 0, -1, -750), (45, 110, 0, 0, 0, -1, -300),
    (90, 90, 1, 0, 0, 3, -750), (96, 88, 0, 0, 0, 20, -750),
])
def test_lane_plan(lane_demo, tmp_path, groups, la, lb, homolog, nolp, stacking, max_diff, opening):
    a = make_rna(la, 31 * la + lb)
    b = make_homolog(a, 7) if homolog else make_rna(lb, 17 * lb + la)
    args = []
    for k, r in enumerate((a, b)):
        f = tmp_path / f"{k}.pp"
        f.write_text(r.to_pp(stacking=bool(stacking)))
        args.append(str(f))
    r = subprocess.run([lane_demo, *args, str(nolp), str(stacking), str(max_diff), str(opening), str(groups)],
                       capture_output=True, text=True, check=True)
    assert r.stdout.startswith("ok "), r.stdout
    if la >= 57 and not nolp:
        assert int(r.stdout.split()[1]) > 1  # several items

"""Index-checking build (libsfac_check.so) on the paths that
tests/test_gpu_check.py does not reach; see tests/check_path_cases.py.  A
failed check records its site and skips the access, so this test faults no GPU
even if a check fires."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def run(oracle_built):
    from ewaldcorrel_b200 import build

    if not os.path.exists(build.LIB_CHECK):
        build.build(check=True)
    env = dict(os.environ, EWALDCORREL_LIBSFAC=build.LIB_CHECK)
    r = subprocess.run([sys.executable, os.path.join(HERE, "check_path_cases.py")], env=env, capture_output=True,
                       text=True, timeout=1200)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_no_index_check_fails(run):
    assert run["library"].endswith("libsfac_check.so") and run["enabled"] == 1 and run["start"][0] == 0
    assert not [c for c in run["cases"] if c["module"] != 0]
    assert len(run["cases"]) == 20


def test_parity(run):
    for c in run["cases"]:
        if "energy_rel" in c:
            assert c["energy_rel"] <= 1e-6 and c["force_rrms"] <= 1e-5 and c["pot_rrms"] <= 1e-5, c


def test_the_failing_launches_failed(run):
    assert run["cases"][-1]["failed"] == 1

"""CMPY_ED_MATVEC is read once per process: the plans made later take the matvec that it named, whatever becomes of the
variable."""

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import os
from cmpy_gb300.models import ChainLattice, HubbardModel
first = HubbardModel(ChainLattice(8, True), inter=4.0, mu=2.0).plan(4, 4)
print(first.matvec_variant)
os.environ.pop("CMPY_ED_MATVEC")
print(HubbardModel(ChainLattice(8, True), inter=3.0, mu=2.0).plan(4, 4).matvec_variant)
"""


@pytest.mark.parametrize("variant", [5, 6, 3])
def test_named_once(cuda, variant):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).resolve().parent.parent, capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, CMPY_ED_MATVEC=str(variant)))
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == [str(variant)] * 2

"""A test that needs the oracle's reference build is skipped where there is no
reference checkout to build it from, and fails where there is one."""
import os
import subprocess
import sys

import pytest

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("where", ["call", "fixture", "highlights"])
@pytest.mark.parametrize("checkout", [False, True])
def test_missing_oracle(tmp_path, where, checkout):
    if oracle.ref_available():
        pytest.skip("the oracle is built")
    body = {"call": "def test_it():\n    oracle.set_threads(1)\n",
            "fixture": "@pytest.fixture\ndef f():\n    oracle.set_threads(1)\n\n\ndef test_it(f):\n    pass\n",
            "highlights": "def test_it():\n    oracle.recover_highlights(np.zeros((8, 8, 3)), 1.0)\n"}[where]
    (tmp_path / "conftest.py").write_text(f"import sys\nsys.path.insert(0, {ROOT!r})\nfrom tests.conftest import *\n")
    (tmp_path / "test_it.py").write_text("import numpy as np\nimport pytest\n\nimport oracle\n\n\n" + body)
    env = dict(os.environ, LRE_REFERENCE_DIR=str(tmp_path / "ref"))
    if checkout:
        (tmp_path / "ref" / "core").mkdir(parents=True)
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider", str(tmp_path)], cwd=tmp_path,
                       env=env, capture_output=True, text=True)
    assert ("1 skipped" in r.stdout) == (not checkout), r.stdout + r.stderr
    assert (r.returncode != 0) == checkout

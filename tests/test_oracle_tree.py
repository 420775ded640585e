"""DISCO_REF names the reference sources that the oracle builds compile: a path
without them is an error, not a silent skip of every oracle build; without
DISCO_REF an absent tree is only absent."""
import os
import subprocess
import sys

import pytest

ORACLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle")


@pytest.mark.parametrize("module", ["pyoracle", "pyc2p"])
def test_wrong_reference_tree_fails(module, tmp_path):
    def load(ref):
        env = {k: v for k, v in os.environ.items() if k != "DISCO_REF"}
        env.update({"DISCO_REF": str(ref)} if ref else {}, PYTHONPATH=ORACLE)
        return subprocess.run([sys.executable, "-c", "import %s as o; print(o.REF_SRC)" % module], env=env,
                              capture_output=True, text=True, timeout=120)
    for wrong in (tmp_path, tmp_path / "none"):
        r = load(wrong)
        assert r.returncode != 0 and "DISCO_REF" in r.stderr, r.stdout
    (tmp_path / "paul.h").write_text("")
    r = load(tmp_path)
    assert r.returncode == 0 and r.stdout.strip() == str(tmp_path)
    assert load(None).returncode == 0

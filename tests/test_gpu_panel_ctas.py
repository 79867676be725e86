"""The blocked reduction on fewer CTAs than a B200 holds (a smaller GPU, or a slice of one): every slot of the panel's
sums has a CTA and a warp, so the eigenvalues are right down to the fewest CTAs whose rows fit."""

import os
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [12, 31, 61, 62, 64, 148])
def test_eigenvalues_on_few_ctas(tmp_path, ctas):
    f = tmp_path / "panel.py"
    f.write_text(textwrap.dedent(f"""
        import sys
        sys.path[:0] = [{str(ROOT / 'am1-rs_b200')!r}]
        import numpy as np
        from am1gpu import native
        for n in (700, 767):
            rng = np.random.default_rng(n)
            a = rng.standard_normal((n, n))
            a = (a + a.T) * 0.5 + np.diag(np.linspace(-3.0, 3.0, n))
            w, ref = native.eigvalsh(a), np.linalg.eigvalsh(a)
            assert np.max(np.abs(w - ref)) < 1e-10 * max(1.0, float(np.max(np.abs(ref)))), n
        print("ok")
    """))
    r = subprocess.run([sys.executable, str(f)], env=dict(os.environ, AM1GPU_BIG="grid", AM1GPU_TRIDIAG_CTAS=str(ctas)), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr

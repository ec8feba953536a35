"""bench.py where the reference library has not been built: the reference arm says so
in one line and ends well."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(os.path.exists(os.path.join(ROOT, 'oracle', '_ref', 'libsprref.so')), reason='the library is built')
def test_reference_arm_without_the_reference():
    r = subprocess.run([sys.executable, 'bench.py', '--impl', 'reference', '--steps', '1', '--warmup', '1'], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line['impl'] == 'reference' and 'not built' in line['unavailable'] and '\n' not in line['unavailable']

"""The autotuners' cached choices hold for the kernels they were measured with."""
from __future__ import annotations

import re
import subprocess
import sys

from conftest import PKG

from test_autotune_rule import _op


def test_version_names_the_kernels_sources():
    from cf_b200 import _lib

    out = subprocess.run([sys.executable, "-c", "import build; print(build.source_id())"], cwd=PKG, capture_output=True,
                         text=True, check=True).stdout.strip()
    assert re.fullmatch(r"[0-9a-f]{12}", out)
    assert out in _lib.version()


def test_keys_change_with_the_version(monkeypatch):
    from cf_b200 import _lib, operator, ragged

    op = _op()
    keys = lambda: (operator._autotune_key(op, 300, "af_sym", operator.AUTOTUNE_PATHS),  # noqa: E731
                    ragged._key([op], [300], ["af_sym"], (0, 4)))
    before = keys()
    monkeypatch.setattr(_lib, "version", lambda: "another")
    after = keys()
    assert before[0] != after[0] and before[1] != after[1]

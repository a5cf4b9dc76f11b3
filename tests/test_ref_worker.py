"""A test that asks for the reference build is skipped where it was not built."""
import unittest

import numpy as np
import pytest


def test_missing_reference_build_skips(monkeypatch, tmp_path):
    import oracle as O
    from oracle.ref_worker import RefWorker
    monkeypatch.setattr(O, "REF_DIR", str(tmp_path))
    with pytest.raises(unittest.SkipTest):
        RefWorker("dirichlet", 4, 1.0, np.ones((5, 5, 5)))

"""A test that asks for the reference's build where there is none is skipped, not failed."""
from __future__ import annotations

import pytest

import oracle


def test_a_missing_reference_build_skips():
    if oracle.ref_available():
        pytest.skip("the build is here")
    oracle.ref()
    raise AssertionError("not reached: ref() raises without the build")


def test_other_missing_files_fail(tmp_path):
    with pytest.raises(FileNotFoundError):
        (tmp_path / "none").read_text()

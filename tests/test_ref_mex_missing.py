"""A comparison with the reference's CUDA code is skipped only where its
sources are not there; with the sources and no library it fails."""
import os
import unittest

import pytest

import ref_mex


@pytest.mark.parametrize("name", sorted(ref_mex.SOURCES))
def test_missing_library_skips_only_without_its_source(name, tmp_path, monkeypatch):
    monkeypatch.setenv("EFIE_REFERENCE_DIR", str(tmp_path))
    monkeypatch.setattr(ref_mex, "REF_DIR", str(tmp_path))
    with pytest.raises(unittest.SkipTest):
        ref_mex.RefMex(name)
    (tmp_path / ref_mex.SOURCES[name]).write_text("")
    with pytest.raises(FileNotFoundError) as e:
        ref_mex.RefMex(name)
    assert not isinstance(e.value, unittest.SkipTest)


def test_sources_are_those_of_the_makefile():
    with open(os.path.join(ref_mex.HERE, "Makefile")) as f:
        make = f.read()
    for name, src in ref_mex.SOURCES.items():
        assert "$(OUT)/%s.so: $(REF)/%s " % (name, src) in make

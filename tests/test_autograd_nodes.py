"""Loader of the autograd nodes: an extension that does not fit gives way to the Python functions, with one warning."""

import warnings

import pytest


@pytest.mark.parametrize("form", ["none", "damaged", "other version"])
def test_extension_that_cannot_be_loaded(monkeypatch, tmp_path, form):
    from returnn_b200.ops import _lib, nodes

    if form == "damaged":
        (tmp_path / nodes.file_name()).write_bytes(b"\x7fELF and no more")
    elif form == "other version":
        (tmp_path / "_autograd_nodes-torch0.1-cpython-20.so").write_bytes(b"not to be opened")
    monkeypatch.setattr(_lib, "_LIB_DIR", str(tmp_path))
    monkeypatch.setattr(nodes, "_module", None)
    monkeypatch.setattr(nodes, "_tried", False)
    with warnings.catch_warnings(record=True) as seen:
        warnings.simplefilter("always")
        assert nodes.active() is None and nodes.active() is None
    assert len(seen) == (0 if form == "none" else 1)
    if seen:
        assert "returnn_b200.ops.build" in str(seen[0].message)

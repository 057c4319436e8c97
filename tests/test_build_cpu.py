"""The oracle's build where the reference's sources are not there."""
from oracle import build as B


def test_reference_kernels_are_optional(tmp_path, monkeypatch):
    for root in (tmp_path, tmp_path / "nowhere"):  # an empty folder, none
        monkeypatch.setattr(B, "REFERENCE_ROOT", str(root))
        monkeypatch.setattr(B, "REF_OUT", str(tmp_path / "_ref"))
        assert B.build_ref_cubins() == []

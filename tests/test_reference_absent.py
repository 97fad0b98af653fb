"""Without the reference's sources, whether their folder is missing or empty, the build goes on without the oracle's
programs."""
from oracle import ref_io


def test_an_empty_folder_is_no_reference(tmp_path):
    for folder in (tmp_path, tmp_path / "missing"):
        assert not ref_io.reference_present(str(folder))
        assert ref_io.build_ref(str(folder)) == ref_io.ref_available()

"""build() where the reference's directory exists but holds no sources."""


def test_build_with_an_empty_reference_directory(lib, tmp_path, monkeypatch):
    import __graft_entry__

    monkeypatch.setenv("SYMX_REFERENCE_DIR", str(tmp_path))
    __graft_entry__.build()

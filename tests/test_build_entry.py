"""build() with and without a reference checkout: the checkers compiled from the
reference's sources are asked for only where those sources are."""
import __graft_entry__ as entry


def test_reference_targets_need_the_sources(tmp_path, monkeypatch):
    asked = []
    monkeypatch.setattr(entry, "_make", lambda directory, *targets: asked.extend(targets))
    monkeypatch.setenv("QWEN_METAL_REF", str(tmp_path))
    entry.build()  # the directory is there, but empty
    assert asked == ["all", "all"]
    (tmp_path / "qwen_host.c").write_text("")
    entry.build()
    assert asked[2:] == ["all", "all", "ref", "ref-test", "ref-bench"]

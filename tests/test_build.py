"""What the build does with what it finds: a reference folder without sources."""
import oracle


def test_an_empty_reference_folder_builds_the_restatement_alone(tmp_path, monkeypatch):
    monkeypatch.setenv("DTCF_REFERENCE", str(tmp_path))
    oracle.build(ref=True)

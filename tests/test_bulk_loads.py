"""The library also runs as one replica per GPU of a node: its bulk loads go to
the loading CTA only."""
import pathlib

CSRC = pathlib.Path(__file__).resolve().parent.parent / "uhm_gb300" / "csrc"


def test_no_bulk_load_to_several_ctas():
    sources = [p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".cpp", ".hpp")]
    assert any("cp.async.bulk.tensor" in p.read_text() for p in sources)
    assert [p.name for p in sources if "multicast::cluster" in p.read_text()] == []

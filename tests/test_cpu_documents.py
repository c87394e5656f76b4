"""Texts of the package that a template was used for."""

import pathlib
import re

ROOT = pathlib.Path(__file__).resolve().parents[1]


def _texts():
    yield from sorted(p for p in ROOT.iterdir() if p.suffix in (".md", ".py"))
    for folder in ("cosmos_predict25_b200", "profiles", "perf", "tests", "scripts", "examples"):
        yield from sorted(p for p in (ROOT / folder).rglob("*") if p.suffix in (".md", ".py", ".cu", ".cuh", ".cpp", ".h") and "_build" not in p.parts)


def test_no_template_marker_is_left_unfilled():
    """A marker for figures to be filled in is two at signs around capitals."""
    marker = re.compile("@" + r"[A-Z][A-Z_]+" + "@")
    texts = list(_texts())
    assert len(texts) > 150
    left = [f"{p.relative_to(ROOT)}:{n}" for p in texts for n, line in enumerate(p.read_text(errors="replace").splitlines(), 1) if marker.search(line)]
    assert left == []

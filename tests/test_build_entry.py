"""build() without the reference sources: an absent or an empty checkout is
passed over, the rest is built."""
import subprocess

import pytest

import __graft_entry__ as entry
from ewaldcorrel_b200 import build as B


@pytest.mark.parametrize("files,refs", [(None, 0), ([], 0), (["sfac.cpp"], 1)])
def test_reference_oracle_only_with_sources(monkeypatch, tmp_path, files, refs):
    ref = tmp_path / "ref"
    if files is not None:
        ref.mkdir()
        for f in files:
            (ref / f).write_text("")
    made = []
    monkeypatch.setattr(entry, "REFERENCE", str(ref))
    monkeypatch.setattr(B, "build", lambda **kw: None)
    monkeypatch.setattr(subprocess, "run", lambda cmd, **kw: made.append(cmd[3]))
    entry.build()
    assert made == ["all"] + ["ref"] * refs

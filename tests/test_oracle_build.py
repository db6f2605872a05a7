"""The oracle's build of the reference: an empty source folder is named, and a
folder whose sources cannot be built is an error, not a silent skip."""
import subprocess

import pytest


def test_empty_folder_is_named(orc, tmp_path, capsys):
    orc.build(ref_src=str(tmp_path))
    assert str(tmp_path) in capsys.readouterr().err


def test_incomplete_folder_is_an_error(orc, tmp_path):
    (tmp_path / "bidiag.c").write_text("")
    with pytest.raises(subprocess.CalledProcessError):
        orc.build(ref_src=str(tmp_path))

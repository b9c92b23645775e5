"""The CPU builds of kernel code are dropped when any kernel header is newer, so an edit of a header
that a fixture does not list (formation_hex.cuh was one) is never tested against an old build."""
import os

import pytest

from conftest import ROOT, drop_stale_emulations


@pytest.mark.parametrize("header", sorted(f for f in os.listdir(os.path.join(ROOT, "cfdv_b200", "csrc"))
                                          if f.endswith((".cuh", ".h"))))
def test_a_newer_header_drops_the_build(tmp_path, header):
    emu, csrc = tmp_path / "emu", tmp_path / "csrc"
    emu.mkdir()
    csrc.mkdir()
    old, new = emu / "libold_emu.so", emu / "libnew_emu.so"
    for p, t in ((csrc / "other.h", 50), (old, 100), (csrc / header, 200), (new, 300), (emu / "src_emu.cpp", 10)):
        p.write_text("")
        os.utime(p, (t, t))
    drop_stale_emulations(str(emu), str(csrc))
    assert not old.exists() and new.exists() and (emu / "src_emu.cpp").exists()

"""Every source file of the library is built."""
import os

from instantgr_b200 import build


def test_every_source_is_in_a_build_list():
    have = {f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cpp"))}
    assert have == {*build.CU_SOURCES, *build.CPP_SOURCES, "main_route.cpp", "gen_main.cpp"}

"""The build refuses a library whose streamed-tile kernels have not the register
count their split needs (a library that has refuses nothing at run time)."""
import os

import pytest

from pdflow import build

LINE = ("ptxas info    : Compiling entry function '_ZN6pdflow3_GLOBAL__N__116k_iterate_streamILb{0}ELb{1}EEEvNS0_10Args' for"
        " 'sm_103a'\nptxas info    : Function properties for x\n    0 bytes stack frame\n"
        "ptxas info    : Used {2} registers, used 2 barriers\n")


def _report(strips=96, tiles=96, direct=128):
    return LINE.format(1, 1, strips) + LINE.format(0, 0, direct) + LINE.format(0, 1, tiles)


def test_the_split_s_count_passes():
    build.check_registers(_report())
    build.check_registers(_report(direct=90))   # no split there


@pytest.mark.parametrize("strips,tiles", [(95, 96), (96, 98), (104, 104)])
def test_another_count_is_refused(strips, tiles):
    with pytest.raises(RuntimeError, match="register"):
        build.check_registers(_report(strips, tiles))


def test_a_report_without_the_kernels_is_refused():
    with pytest.raises(RuntimeError, match="report"):
        build.check_registers(LINE.format(0, 0, 96))


def test_the_built_library_passes(built_lib):
    build.check_registers(open(os.path.join(build.LIBDIR, "ptxas.log")).read())

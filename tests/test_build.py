"""The build gives the same kernels every time: a file of several kernels
compiled side by side comes out at one size (names of temporary files apart)."""
import concurrent.futures as cf

from gaffa_b200 import build


def test_compilation_is_repeatable(tmp_path):
    def size(k):
        obj = tmp_path / f"{k}.o"
        build._compile(build.CSRC / "dedisperse_mma.cu", obj)
        return obj.stat().st_size

    with cf.ThreadPoolExecutor(4) as ex:
        assert len(set(ex.map(size, range(4)))) == 1

"""What skips a test and what does not."""
import pytest

from oracle import ref_cpu

pytest_plugins = ["pytester"]


def test_only_the_missing_oracle_skips(pytester, request):
    conftest = request.config.rootpath / "tests" / "conftest.py"
    pytester.makeconftest(f"import sys\nsys.path.insert(0, {str(request.config.rootpath)!r})\n" + conftest.read_text())
    pytester.makepyfile("""
        import ctypes
        def test_library_that_does_not_load():
            ctypes.CDLL("/nonexistent/library.so")
        def test_oracle():
            from oracle import ref_cpu
            ref_cpu.max_threads()
    """)
    result = pytester.runpytest_inprocess("-p", "no:cacheprovider")
    result.assert_outcomes(failed=1, **({"passed": 1} if ref_cpu.available() else {"skipped": 1}))

"""A test kernel is built again when its source or a header of the package is newer than what was built."""
import os

import __graft_entry__ as entry
import conftest


def test_older_than_a_header(tmp_path, monkeypatch):
    from tqllm_b200 import build
    header, built = tmp_path / "h.cuh", tmp_path / "quotient_kernel.so"
    source = os.path.join(entry.ROOT, "tests", "quotient_kernel.cu")
    calls = []
    monkeypatch.setattr(build, "_deps", lambda: [str(header)])
    monkeypatch.setattr(entry, "TEST_KERNELS", ("quotient_kernel",))
    monkeypatch.setattr(entry, "kernel_path", lambda name: str(built))
    monkeypatch.setattr(entry, "build_test_kernel", calls.append)
    refresh = conftest.current_test_kernels.__wrapped__
    header.write_text("")
    refresh()                                             # nothing was built: the tests that need it build it
    assert not calls and not entry.kernel_is_current("quotient_kernel")
    built.write_text("")
    now = os.path.getmtime(source) + 100
    os.utime(header, (now, now))
    os.utime(built, (now + 1, now + 1))
    refresh()
    assert not calls
    os.utime(header, (now + 2, now + 2))
    refresh()
    assert calls == ["quotient_kernel"]

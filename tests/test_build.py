"""The build's own decisions, with the compilers replaced by a recorder (no GPU, nothing is compiled)."""
import os
import sysconfig

from juliavision_b200 import _lib, build


def test_the_native_host_side_is_built_per_interpreter():
    """It is compiled against one interpreter's headers: its name says which, so that another finds none and builds its own."""
    assert os.path.basename(_lib.HOST_PATH) == "hostcalls" + sysconfig.get_config_var("EXT_SUFFIX")
    assert os.path.normpath(build.HOST_SO) == os.path.normpath(_lib.HOST_PATH)


def test_the_library_is_linked_before_the_host_side_can_fail(monkeypatch):
    """Without Python's headers the extension does not compile; the C-ABI library is there all the same."""
    ran = []
    monkeypatch.setattr(build, "_stale", lambda target, deps: target in (build.SO, build.HOST_SO))
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: ran.append(cmd[cmd.index("-o") + 1]))
    build.build()
    assert ran == [build.SO, build.HOST_SO]

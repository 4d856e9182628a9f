"""CPU: the native call path belongs to the interpreter it was built for."""
import os
import sysconfig

import build
import lbcube as E


def test_module_is_named_for_this_interpreter():
    """Another Python neither finds this one's module nor keeps it as up to date."""
    tag = sysconfig.get_config_var("EXT_SUFFIX")
    assert os.path.basename(E.CALL_PATH) == os.path.basename(build.CALL) == "_lbcall" + tag

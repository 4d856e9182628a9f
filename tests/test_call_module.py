"""CPU: the native call path belongs to the interpreter it was built for, and takes
ints of a class of their own (as ctypes does) as addresses."""
import enum
import os
import sysconfig

import pytest

import build
import lbcube as E
from test_call_path import A, CALLS


class Address(enum.IntEnum):
    BUFFER = A[0]
    STREAM = 0


def test_module_is_named_for_this_interpreter():
    """Another Python neither finds this one's module nor keeps it as up to date."""
    tag = sysconfig.get_config_var("EXT_SUFFIX")
    assert os.path.basename(E.CALL_PATH) == os.path.basename(build.CALL) == "_lbcall" + tag


@pytest.mark.parametrize("name", sorted(CALLS))
@pytest.mark.parametrize("args", [{"p": Address.BUFFER}, {"p": True}, {"s": Address.STREAM}], ids=str)
def test_int_subclasses_as_addresses(name, args, monkeypatch):
    """Fake addresses: every call is refused by the launcher's validation."""
    E.load()
    if "s" in args and name.startswith("launch"):
        pytest.skip("no stream argument")
    native = CALLS[name](**args)
    monkeypatch.setattr(E, "_call", None)
    assert native == CALLS[name](**args) == E.cudaErrorInvalidValue

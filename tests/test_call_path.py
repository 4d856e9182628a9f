"""CPU: the native call path of the step launchers (csrc/pycall.c) against the
ctypes path. Both must return the same status for the same arguments, and
whatever the native path does not take (it returns None) must reach ctypes and
be accepted or refused there as before. Fake, never-dereferenced addresses:
every call is rejected by the launcher's validation before any CUDA call."""
import os

import numpy as np
import pytest

import lbcube as E

A = [0x10000000 * k for k in range(1, 8)]

CALLS = {
    "step_async": lambda **k: E.step_async(k.get("lat", "D3Q19"), k.get("real", "float"), "TRT", k.get("p", A[0]), A[1],
                                           k.get("nx", 0), 8, 8, k.get("w", 1.5), k.get("s")),
    "launch_step_gpu": lambda **k: E.launch_step_gpu(k.get("lat", "D3Q19"), k.get("real", "float"), "TRT", k.get("p", A[0]),
                                                     A[1], k.get("nx", 0), 8, 8, k.get("w", 1.5)),
    "step_shifted_async": lambda **k: E.step_shifted_async(k.get("lat", "D3Q19"), "f16s", "MRT", k.get("p", A[0]), A[1],
                                                           k.get("nx", 0), 8, 8, k.get("w", 1.5), stream=k.get("s")),
    "scalar_step_async": lambda **k: E.scalar_step_async(k.get("lat", "D3Q19"), k.get("real", "float"), k.get("p", A[0]),
                                                         A[1], A[2], k.get("nx", 0), 8, 8, k.get("w", 1.5),
                                                         stream=k.get("s")),
    "launch_scalar_step_gpu": lambda **k: E.launch_scalar_step_gpu(k.get("lat", "D3Q19"), k.get("real", "float"),
                                                                   k.get("p", A[0]), A[1], A[2], k.get("nx", 0), 8, 8,
                                                                   k.get("w", 1.5)),
    "reaction_ab_async": lambda **k: E.reaction_ab_async(k.get("lat", "D3Q19"), k.get("real", "float"), k.get("p", A[0]),
                                                         A[1], A[2], A[3], A[4], k.get("nx", 0), 8, 8, k.get("w", 1.5),
                                                         0.1, k.get("s")),
    "launch_reaction_AB_gpu": lambda **k: E.launch_reaction_AB_gpu(k.get("lat", "D3Q19"), k.get("real", "float"),
                                                                   k.get("p", A[0]), A[1], A[2], A[3], A[4],
                                                                   k.get("nx", 0), 8, 8, k.get("w", 1.5), 0.1),
    "fluid_reaction_ab_async": lambda **k: E.fluid_reaction_ab_async(
        k.get("lat", "D3Q19"), k.get("real", "float"), "MRT", k.get("p", A[0]), A[1], A[2], A[3], A[4], A[5],
        k.get("nx", 0), 8, 8, k.get("w", 1.5), 1.2, 0.1, stream=k.get("s")),
}


class Buffer:
    def __init__(self, address):
        self.address = address

    def data_ptr(self):
        return self.address


class Stream:
    cuda_stream = 0


ARGS = [{}, {"p": None}, {"p": Buffer(A[0])}, {"p": Buffer(A[1]), "nx": 8}, {"nx": 2 ** 40}, {"nx": -1}, {"nx": True, "p": None},
        {"w": 1}, {"w": np.float64(1.5)}, {"lat": "D2Q9", "nx": 0}, {"s": 0}, {"s": Stream()}, {"real": "double"},
        {"lat": "D2Q5"}, {"lat": "nonsense"}, {"real": "half"}, {"p": "text"}, {"nx": 1.5}, {"w": "x"}]


@pytest.mark.parametrize("name", sorted(CALLS))
@pytest.mark.parametrize("args", ARGS, ids=str)
def test_same_outcome_as_ctypes(name, args, monkeypatch):
    E.load()
    if E._call is None:
        pytest.skip("built without the Python headers")
    if "s" in args and name.startswith("launch"):
        pytest.skip("no stream argument")

    def outcome():
        try:
            return CALLS[name](**args)
        except Exception as e:  # noqa: BLE001
            return type(e).__name__

    native = outcome()
    monkeypatch.setattr(E, "_call", None)
    assert native == outcome()


def test_plain_arguments_take_the_native_path():
    E.load()
    if E._call is None:
        assert not os.path.exists(E.CALL_PATH)
        return
    assert E._call.step("D3Q19", "float", "TRT", None, A[1], 8, 8, 8, 1.5, None) == E.cudaErrorInvalidDevicePointer
    assert E._call.step("D3Q19", "float", "TRT", None, A[1], 8, 8, 8, 1, None) is None  # an int rate: ctypes
    with pytest.raises(TypeError):
        E._call.step("D3Q19", "float")

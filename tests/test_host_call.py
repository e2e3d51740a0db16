"""Calls of launchers without ctypes (csrc/host_call.cu): arguments arrive as ctypes hands them over, whatever their number and
order; what is no number or address is refused."""

from __future__ import annotations

import ctypes
import random
import shutil
import subprocess
import threading

import pytest

KINDS = {"i": ("int", ctypes.c_int), "l": ("long", ctypes.c_long), "p": ("void*", ctypes.c_void_p), "f": ("float", ctypes.c_float)}


@pytest.fixture(scope="module")
def callees(tmp_path_factory):
    """Functions of many signatures that put their arguments, as text, into a buffer."""
    compiler = shutil.which("gcc") or shutil.which("cc")
    if compiler is None:
        pytest.skip("no C compiler")
    rng = random.Random(5)
    signatures = ["", "i", "f", "p", "iiiiiii", "ffffffff", "pifl" * 8] + [
        "".join(rng.choice("iilppp") for _ in range(rng.randint(1, 48))) for _ in range(12)]
    for k, s in enumerate(signatures[7:]):  # floats at odd places, eight at most
        for _ in range(k % 9):
            at = rng.randrange(len(s) + 1)
            s = s[:at] + "f" + s[at:]
        signatures[7 + k] = s
    source = "#include <stdio.h>\nchar seen[4096];\n"
    for n, s in enumerate(signatures):
        source += f"int f{n}({', '.join(f'{KINDS[k][0]} a{i}' for i, k in enumerate(s)) or 'void'}) {{ char* p = seen; *p = 0;\n"
        for i, k in enumerate(s):
            source += f'p += sprintf(p, "{dict(i="%d", l="%ld", p="%p", f="%a")[k]} ", a{i});\n'
        source += f"return {n} - 3; }}\n"
    folder = tmp_path_factory.mktemp("callees")
    (folder / "c.c").write_text(source)
    subprocess.run([compiler, "-O2", "-w", "-shared", "-fPIC", str(folder / "c.c"), "-o", str(folder / "c.so")], check=True)
    lib = ctypes.CDLL(str(folder / "c.so"))
    made = []
    for n, s in enumerate(signatures):
        fn = getattr(lib, f"f{n}")
        fn.argtypes, fn.restype = [KINDS[k][1] for k in s], ctypes.c_int
        made.append((s, fn))
    return made, ctypes.c_char.in_dll(lib, "seen")


def _native(fn):
    from qwen3_runtime_b200.ops import build

    made = build.native_caller(fn)
    if made is fn:
        pytest.skip("no native calls on this machine")
    return made


def _values(signature, rng):
    draw = dict(i=lambda: rng.choice([0, 1, -1, 2 ** 31 - 1, -2 ** 31, rng.randint(-9, 9)]),
                f=lambda: rng.choice([0.0, -1.5, 3, 1e30, 0.1]), l=lambda: rng.choice([0, -1, 2 ** 62, -2 ** 62, 5]),
                p=lambda: rng.choice([None, 1, 2 ** 47 - 8, rng.getrandbits(46)]))
    return [draw[k]() for k in signature]


def test_arguments_arrive_as_through_ctypes(callees):
    rng = random.Random(1)
    functions, seen = callees
    for signature, fn in functions:
        native = _native(fn)
        for _ in range(6):
            values = _values(signature, rng)
            code = fn(*values)
            want = ctypes.string_at(ctypes.addressof(seen))
            assert native(*values) == code and ctypes.string_at(ctypes.addressof(seen)) == want, signature


def test_what_is_no_argument_is_refused(callees):
    by_signature = dict(callees[0])
    native = _native(by_signature["iiiiiii"])
    for bad in ((1, 2, 3), (1,) * 8, (1, 2, 3, 4, 5, 6, None), (1, 2, 3, 4, 5, 6, 1.0), (1, 2, 3, 4, 5, 6, "7")):
        with pytest.raises(TypeError):
            native(*bad)
    with pytest.raises(OverflowError):
        native(1, 2, 3, 4, 5, 6, 1 << 70)
    with pytest.raises(TypeError):
        _native(by_signature["f"])("x")
    with pytest.raises(TypeError):
        _native(by_signature["p"])(1.5)


def test_what_stands_for_a_whole_number_is_taken_as_ctypes_takes_it(callees):
    numpy, torch = pytest.importorskip("numpy"), pytest.importorskip("torch")

    class Stands:
        def __index__(self):
            return -7

    class Refuses:
        def __index__(self):
            raise ValueError("none")

    by_signature, seen = dict(callees[0]), callees[1]
    fn = by_signature["iiiiiii"]
    native = _native(fn)
    values = (True, numpy.int64(5), numpy.uint8(200), torch.tensor(-3), torch.tensor([9]), Stands(), numpy.int32(-2 ** 31))
    code = fn(*values)
    want = ctypes.string_at(ctypes.addressof(seen))
    assert native(*values) == code and ctypes.string_at(ctypes.addressof(seen)) == want
    with pytest.raises(ValueError):
        native(1, 2, 3, 4, 5, 6, Refuses())
    for bad in (numpy.float64(2), torch.tensor(1.5), torch.tensor([1, 2])):
        with pytest.raises(ctypes.ArgumentError):
            fn(1, 2, 3, 4, 5, 6, bad)
        with pytest.raises(TypeError):
            native(1, 2, 3, 4, 5, 6, bad)
    address = by_signature["p"]
    with pytest.raises(ctypes.ArgumentError):
        address(numpy.int64(8))
    with pytest.raises(TypeError):
        _native(address)(numpy.int64(8))


def test_signatures_beyond_the_common_type_stay_with_ctypes(callees):
    from qwen3_runtime_b200.ops import build

    fn = callees[0][0][1]
    _native(fn)
    for types in ([ctypes.c_int] * 49, [ctypes.c_float] * 9, [ctypes.c_double]):
        other = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *a: 0)
        other.argtypes, other.restype = types, ctypes.c_int
        assert build.native_caller(other) is other


def test_every_launcher_is_called_natively():
    from qwen3_runtime_b200.ops import build
    from qwen3_runtime_b200.ops.cuda import _SIGNATURES

    for names in _SIGNATURES.values():
        for types in names.values():
            assert all(t in build._KINDS for t in types)
            assert sum(t is ctypes.c_float for t in types) <= 8 and len(types) <= 48


def test_threads_call_at_the_same_time(callees):
    native = _native(dict(callees[0])["i"])
    wrong = []

    def work():
        wrong.extend(1 for _ in range(2000) if native(3) != -2)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

"""CPU: the C-ABI library loads and exports every symbol include/b2l.h declares; the
ctypes structure mirrors have the layout a C compiler gives the header's structs."""
import ctypes as C
import os
import re
import subprocess

import pytest

import __graft_entry__ as entry

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "b2l.h")


@pytest.fixture(scope="module")
def L():
    entry.build()
    from lit_llama_b200 import _lib

    return _lib


def declared_functions():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(b2l_[a-z0-9_]+)\s*\(", src)))


def test_every_declared_symbol_is_exported_and_bound(L):
    names = declared_functions()
    assert len(names) >= 20
    handle = C.CDLL(L.LIB_PATH)
    for n in names:
        assert hasattr(handle, n), f"{n} declared in b2l.h but not exported"
    assert sorted(L.EXPORTS) == names, "ctypes binding and header disagree"
    assert L.lib().b2l_version() == 100


def test_struct_layout_matches_c_compiler(L, tmp_path):
    prog = tmp_path / "layout.c"
    prog.write_text(
        '#include <stdio.h>\n#include <stddef.h>\n#include "b2l.h"\n'
        "int main(void){\n"
        'printf("%zu %zu %zu %zu\\n", sizeof(b2l_q4_linear_args), sizeof(b2l_q4_weight), sizeof(b2l_layer), sizeof(b2l_decode_args));\n'
        'printf("%zu %zu %zu\\n", offsetof(b2l_q4_linear_args, flags), offsetof(b2l_layer, k_cache), offsetof(b2l_decode_args, logits));\n'
        "return 0;}\n")
    exe = tmp_path / "layout"
    subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(prog), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    got = [C.sizeof(L.Q4LinearArgs), C.sizeof(L.Q4Weight), C.sizeof(L.Layer), C.sizeof(L.DecodeArgs),
           L.Q4LinearArgs.flags.offset, L.Layer.k_cache.offset, L.DecodeArgs.logits.offset]
    assert [int(v) for v in out] == got


def test_errors_are_reported_not_swallowed(L):
    lib = L.lib()
    rc = lib.b2l_q_linear(None, 0, None, None, None, 0, None, None, 0, 1, 1, 2, 4, 2, None)
    assert rc == -1 and b"null pointer" in lib.b2l_last_error()
    assert lib.b2l_q4_tiled_bytes(128, 64) == 128 * 64 // 2
    assert lib.b2l_q4_tiled_bytes(130, 64) == 256 * 64 // 2  # rows padded to a multiple of 128
    assert lib.b2l_q4_tiled_bytes(128, 48) == 0              # K must be a multiple of 32
    assert lib.b2l_decode_step(None, None) == -1
    # tensor-parallel exchange: buffer size = 2 epoch parities x world senders x n/2 words of 8 bytes; bad arguments say so
    assert lib.b2l_tp_buffer_bytes(2, 4096) == 2 * 2 * 2048 * 8
    assert lib.b2l_tp_buffer_bytes(9, 4096) == 0 and lib.b2l_tp_buffer_bytes(2, 4095) == 0
    assert lib.b2l_tp_allreduce(None, None, None, 0, 0, None) == -1 and b"null pointer" in lib.b2l_last_error()
    comm = L.TPComm()
    comm.rank, comm.world, comm.max_elems = 3, 2, 4096
    assert lib.b2l_tp_allreduce(C.byref(comm), C.c_void_p(16), C.c_void_p(16), 4096, 0, None) == -1
    assert b"bad rank" in lib.b2l_last_error()


def test_the_extension_is_optional_and_never_built_by_a_call(L, monkeypatch):
    """Without csrc/pycall.cpp's file the same functions are called through ctypes, with the same answers; no compiler runs for it, however new the headers."""
    from lit_llama_b200 import _build

    handle, built = L.lib(), L.pycall
    calls = [("q4", (which, None, 64, None, None, None, 0, None, 1, 1, 1, 64, None, 0)) for which in range(4)] + [("q8", (None, 64, None, None, None, 1, None, 2, 1, 64, 6.0, 0))]
    answers = [getattr(built, n)(*a) for n, a in calls]
    assert all(a != 0 for a in answers)
    monkeypatch.setenv("NVCC", "/nonexistent/nvcc")
    monkeypatch.setitem(_build.LIBRARIES["pycall"], "out", "/nonexistent/_pycall.abi3.so")
    try:
        L._bind(handle)
        assert isinstance(L.pycall, L._Foreign) and [getattr(L.pycall, n)(*a) for n, a in calls] == answers
    finally:
        monkeypatch.undo()
        L._bind(handle)
    assert type(L.pycall) is type(built)
    assert _build._headers(_build.LIBRARIES["pycall"]) == [HEADER] and _build.LIBRARIES["pycall"]["out"].endswith(".abi3.so")


def test_sequence_functions_take_what_ctypes_takes(monkeypatch):
    """csrc/seqcall.cpp's functions against the ctypes functions they stand for: the same answers and messages for arguments that convert, that ctypes truncates
    or unwraps, and the same refusals; without the file, and with another signature, ctypes'.  No call gets as far as a launch."""
    from lit_llama_b200 import _build
    from lit_llama_b200 import _seqlib as S

    lib, handle = S.lib(), C.CDLL(_build.LIBRARIES["seq"]["out"])
    made = [n for n in S.EXPORTS if type(getattr(lib, n)).__name__ == "builtin_function_or_method"]
    if not os.path.exists(_build.LIBRARIES["seqcall"]["out"]):
        assert not made
        pytest.skip("the extension is not built")
    assert len(made) == sum(S._SIGS[n][0] is C.c_int and bool(S._SIGS[n][1]) and all(a in (C.c_void_p, C.c_int, C.c_float, C.c_longlong, C.c_size_t) for a in S._SIGS[n][1])
                            for n in S.EXPORTS if n not in ("b2l_seq_scan_chunks", "b2l_seq_latent_attention_warps", "b2l_seq_mingru_chunks"))
    for n in made:
        slow, (slow.restype, slow.argtypes) = getattr(handle, n), S._SIGS[n]

        def outcome(f, args):
            try:
                return f(*args), lib.b2l_seq_last_error()
            except (TypeError, C.ArgumentError) as e:
                return type(e)

        args = [None if a is C.c_void_p else 0.5 if a is C.c_float else 0 for a in S._SIGS[n][1]]
        first, ints = S._SIGS[n][1].index(C.c_void_p), [i for i, a in enumerate(S._SIGS[n][1]) if a is C.c_int]
        calls = [args, args[:-1], args + [0], [C.c_void_p(None) if i == first else a for i, a in enumerate(args)], ["x" if i == first else a for i, a in enumerate(args)]]
        for v in (-1, True, 2 ** 31 - 1, 2 ** 32, -2 ** 40, 2 ** 70, 1.0, None):
            calls.append([v if ints and i == ints[-1] else a for i, a in enumerate(args)])
        calls.append([1 if a == 0.5 else a for a in args])
        for c in calls:
            assert outcome(getattr(lib, n), c) == outcome(slow, c), (n, c)
        with pytest.raises(TypeError):
            getattr(lib, n)(*args[:-1], stream=0)
    monkeypatch.setitem(S._SIGS, "b2l_seq_norm", (C.c_int, S._SIGS["b2l_seq_norm"][1] + [C.c_int]))
    assert type(S._functions(handle).b2l_seq_norm) is not type(lib.b2l_seq_norm)
    monkeypatch.setitem(_build.LIBRARIES["seqcall"], "out", "/nonexistent/_seqcall.abi3.so")
    assert type(S._functions(handle).b2l_seq_rope) is not type(lib.b2l_seq_rope)

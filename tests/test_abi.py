"""CPU tests of the C-ABI boundary: the library loads, exports every declared symbol, and rejects bad
arguments on the host without touching a GPU."""
import ctypes as C
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge
    ge.build()
    from kda_b200 import _lib
    return _lib.load()


def test_exports_every_declared_symbol(lib):
    import __graft_entry__ as ge
    names = ge.declared_symbols()
    assert {"kda_recurrent_fwd", "kda_chunk_fwd", "kda_chunk_bwd", "kda_b200_strerror"} <= set(names)
    for n in names:
        assert hasattr(lib, n), n


def test_exports_nothing_but_the_declared_symbols(lib):
    """The header says its entries are the library's only exports: development checks live in libkda_b200_debug.so."""
    import subprocess
    import __graft_entry__ as ge
    from kda_b200 import _lib
    out = subprocess.run(["nm", "-D", "--defined-only", _lib.LIB_PATH], capture_output=True, text=True, check=True).stdout
    exported = {ln.split()[-1] for ln in out.splitlines() if " T " in ln}
    assert exported == set(ge.declared_symbols()) == set(_lib.EXPORTS)


def test_version_and_error_text(lib):
    import re
    from kda_b200 import _lib
    header = open(os.path.join(ROOT, "include", "kda_b200.h")).read()
    assert lib.kda_b200_abi_version() == int(re.search(r"#define KDA_B200_ABI_VERSION (\d+)", header).group(1)) == _lib.ABI_VERSION
    assert lib.kda_b200_strerror(0) == b"ok"
    assert b"NULL" in lib.kda_b200_strerror(-1)
    assert b"workspace" in lib.kda_b200_strerror(-5)
    assert b"tensor map" in lib.kda_b200_strerror(-8)
    assert lib.kda_chunk_status(None, None) == -1


def test_workspace_sizes_are_monotone(lib):
    a = lib.kda_chunk_workspace_bytes(4096, 1, 2, 128, 128, 0)
    b = lib.kda_chunk_workspace_bytes(4096, 1, 2, 128, 128, 1)
    c = lib.kda_chunk_workspace_bytes(8192, 1, 2, 128, 128, 1)
    assert 0 < a < b < c
    assert lib.kda_chunk_max_chunks(130, 2) == 4
    assert lib.kda_chunk_bwd_workspace_bytes(4096, 1, 2, 128, 128, 0) > 0


def test_argument_errors_without_gpu(lib):
    from kda_b200 import _lib
    assert lib.kda_recurrent_fwd(None, None) == -1
    assert lib.kda_chunk_fwd(None, None) == -1
    r = _lib.RecurrentArgs(N=1, T=4, tokens=4, H=2, K=48, V=64, io_dtype=0)
    r.q = r.k = r.v = r.g = r.beta = r.o = C.c_void_p(256)
    assert lib.kda_recurrent_fwd(C.byref(r), None) == -2          # K = 48 unsupported
    r.K = 64
    r.io_dtype = 7
    assert lib.kda_recurrent_fwd(C.byref(r), None) == -3          # dtype
    r.io_dtype = 0
    r.q = C.c_void_p(260)
    assert lib.kda_recurrent_fwd(C.byref(r), None) == -4          # alignment
    r.q = C.c_void_p(0)
    assert lib.kda_recurrent_fwd(C.byref(r), None) == -1          # NULL
    a = _lib.ChunkArgs(tokens=64, N=1, H=2, K=64, V=64, io_dtype=0)
    assert lib.kda_chunk_fwd(C.byref(a), None) == -2              # K, V must be 128
    a.K = a.V = 128
    assert lib.kda_chunk_fwd(C.byref(a), None) == -1              # NULL pointers
    a.q = a.k = a.v = a.g = a.beta = a.o = a.cu_seqlens = a.workspace = C.c_void_p(512)
    a.workspace_bytes = 16
    assert lib.kda_chunk_fwd(C.byref(a), None) == -5              # workspace too small


def test_recurrent_backward_refuses_unaligned_pointers(lib):
    """Loads and stores that are 16 bytes wide: an odd address is an argument error on the host, never a launch."""
    from kda_b200 import _lib
    size = lib.kda_recurrent_bwd_workspace_bytes(64, 1, 2, 64, 64)
    names = ("q", "k", "v", "g", "h0", "d_o", "d_ht", "dq", "dk", "dv", "dg", "dh0")
    for odd in ("v", "h0", "d_o", "d_ht", "dv", "dh0"):
        r = _lib.RecurrentBwdArgs(N=1, T=64, tokens=64, H=2, K=64, V=64, HQ=2, io_dtype=_lib.KDA_FP32, beta=256, dbeta=256, workspace=512, workspace_bytes=size,
                                  **{n: 256 + (4 if n == odd else 0) for n in names})
        assert lib.kda_recurrent_bwd(C.byref(r), None) == -4, odd


def test_kernels_chained_to_the_callers_use_no_read_only_loads():
    """A decode kernel is launched as a programmatic dependent of whatever the caller ran before: it may be brought up while that kernel still
    writes q, k, v, g, beta.  Read-only loads (__ldg, ld.global.nc, const __restrict__ parameters) are undefined for such data."""
    import re
    csrc = os.path.join(ROOT, "kda_b200", "csrc")
    for name in ("kda_decode_bulk.cu", "kda_recurrent.cu"):
        text = open(os.path.join(csrc, name)).read()
        assert "launch_chained" in text and "chain_point();" in text, name
        code = re.sub(r"//[^\n]*", "", text)
        for word in ("__ldg", "ld.global.nc", "__restrict__"):
            assert word not in code, (name, word)
    loaders = open(os.path.join(csrc, "kda_common.cuh")).read()
    assert "__ldg" not in re.sub(r"//[^\n]*", "", loaders)


def _header_fields(struct):
    """(name, ctype) of a struct of the public header, in order."""
    import re
    text = open(os.path.join(ROOT, "include", "kda_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (struct, struct), text, flags=re.S).group(1)
    kinds = {"int32_t": C.c_int32, "int64_t": C.c_int64, "size_t": C.c_size_t, "float": C.c_float}
    out = []
    for decl in filter(None, (d.strip() for d in body.split(";"))):
        kind, names = re.match(r"(?:const\s+)?(\w+)\s*(.*)", decl, flags=re.S).groups()
        for n in names.split(","):
            out.append((n.strip(" *\n"), C.c_void_p if "*" in n else kinds[kind]))
    return out


def test_bindings_have_the_headers_fields(lib):
    """The ctypes structs of the package, and the binding that the integration document gives a maintainer to copy, list the header's fields in
    the header's order: a struct that ends early makes the library read whatever lies behind it."""
    import re
    from kda_b200 import _lib
    for struct, cls in (("kda_recurrent_args", _lib.RecurrentArgs), ("kda_recurrent_bwd_args", _lib.RecurrentBwdArgs), ("kda_chunk_args", _lib.ChunkArgs),
                        ("kda_gate_args", _lib.GateArgs)):
        assert list(cls._fields_) == _header_fields(struct), struct
    doc = open(os.path.join(ROOT, "INTEGRATION.md")).read()
    code = re.search(r"class ChunkArgs\(C\.Structure\):.*?(?=\n\n)", doc, flags=re.S).group(0)
    scope = {"C": C}
    exec(code, scope)      # the class statement of the document
    assert list(scope["ChunkArgs"]._fields_) == _header_fields("kda_chunk_args")
    assert "kda_b200_abi_version() == %d" % _lib.ABI_VERSION in doc


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from kda_b200 import _lib
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "absent.so"))
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _lib.load()


def test_training_pair_refuses_what_it_does_not_take(lib):
    """kda_recurrent_train_fwd / _bwd: argument errors on the host, nothing launched."""
    from kda_b200 import _lib
    size = lib.kda_recurrent_saved_bytes(64, 1, 2, 64, 64)
    assert 0 < size < lib.kda_recurrent_bwd_workspace_bytes(64, 1, 2, 64, 64)
    ok = dict(q=256, k=256, v=256, g=256, beta=256, o=256, N=1, T=64, tokens=64, H=2, K=64, V=64, HQ=2, io_dtype=_lib.KDA_FP32)
    call = lambda saved=256, n=size, **kw: lib.kda_recurrent_train_fwd(C.byref(_lib.RecurrentArgs(**{**ok, **kw})), saved, n, None)      # noqa: E731
    assert call(K=96) == -2 and call(V=256) == -2 and call(tokens=63) == -2
    assert call(h0=512, ht=512) == -2 and call(transpose_state=1) == -2 and call(A_log=256) == -2 and call(beta_sigmoid=1) == -2
    assert call(state_indices=256) == -2
    assert call(io_dtype=_lib.KDA_BF16) == -3
    assert call(saved=None) == -1 and call(o=None) == -1
    assert call(n=size - 1) == -5
    assert call(saved=264) == -4 and call(v=260) == -4 and call(ht=264) == -4 and call(q=260) == -4
    bwd = dict(q=256, k=256, v=256, g=256, beta=256, d_o=256, dq=256, dk=256, dv=256, dg=256, dbeta=256, N=1, T=64, tokens=64, H=2, K=64, V=64, HQ=2,
               io_dtype=_lib.KDA_FP32, workspace=256, workspace_bytes=lib.kda_recurrent_bwd_workspace_bytes(64, 1, 2, 64, 64) - size)
    back = lambda saved=256, n=size, **kw: lib.kda_recurrent_train_bwd(C.byref(_lib.RecurrentBwdArgs(**{**bwd, **kw})), saved, n, None)      # noqa: E731
    assert back(saved=None) == -1 and back(n=size - 1) == -5 and back(saved=272) == -4
    assert back(workspace_bytes=bwd["workspace_bytes"] - 1) == -5 and back(d_o=260) == -4
    assert lib.kda_recurrent_bwd(C.byref(_lib.RecurrentBwdArgs(**bwd)), None) == -5      # without the saved states the workspace holds them too


def test_walk_forward_refuses_what_the_training_forward_refuses(lib):
    """kda_recurrent_walk_fwd: the checks of kda_recurrent_train_fwd, without a buffer to leave anything in."""
    from kda_b200 import _lib
    ok = dict(q=256, k=256, v=256, g=256, beta=256, o=256, N=1, T=64, tokens=64, H=2, K=64, V=64, HQ=2, io_dtype=_lib.KDA_FP32)
    call = lambda **kw: lib.kda_recurrent_walk_fwd(C.byref(_lib.RecurrentArgs(**{**ok, **kw})), None)      # noqa: E731
    assert call(K=96) == -2 and call(tokens=63) == -2 and call(h0=512, ht=512) == -2 and call(transpose_state=1) == -2 and call(A_log=256) == -2
    assert call(io_dtype=_lib.KDA_BF16) == -3 and call(o=None) == -1 and call(v=260) == -4 and call(q=260) == -4


def _bwd_args(**kw):
    from kda_b200 import _lib
    a = dict(q=256, k=256, v=256, g=256, beta=256, d_o=256, dq=256, dk=256, dv=256, dg=256, dbeta=256, N=8, T=2048, tokens=16384, H=32, K=128, V=128,
             HQ=32, io_dtype=_lib.KDA_FP32, workspace=256)
    return _lib.RecurrentBwdArgs(**{**a, **kw})


def test_float32_backward_scratch_holds_what_the_call_needs(lib):
    """kda_recurrent_bwd_scratch_bytes: two rows per token for per-value-head dq, dk only with grouped heads or normalised rows, norms only with
    normalised rows, copies of h0 and d_ht only where dh0 overlaps them, and no states per sequence."""
    size = lambda saved=0, passes=1, **kw: lib.kda_recurrent_bwd_scratch_bytes(C.byref(_bwd_args(**kw)), saved, passes)      # noqa: E731
    rows, states = 16384 * 32 * 128 * 4, 8 * 32 * 128 * 128 * 4
    assert size() < 16384 // 32 * 32 * 65536 * 2 + 1.2 * rows                 # the kept states and r, dbeta's parts
    assert size(use_qk_l2norm=1) - size() == 2 * rows + 16384 * 32 * 8
    assert size(HQ=8) - size() == 2 * rows
    assert size(h0=256, d_ht=1 << 40, dh0=1 << 45) == size()
    assert size(d_ht=1 << 40, dh0=1 << 40) - size() == size(h0=(1 << 40) + states - 16, dh0=1 << 40) - size() == states
    assert size(h0=(1 << 40) + states, dh0=1 << 40) == size()
    assert size(1) == size() - 16384 // 32 * 32 * 65536 - rows
    assert size(N=2000, T=5, tokens=10000, H=8, HQ=8) < 10000 * 8 * (2048 * 2 + 512 + 32) + 4096
    # the upper bound covers every call
    bound = lib.kda_recurrent_bwd_workspace_bytes(16384, 8, 32, 128, 128)
    assert bound == size(use_qk_l2norm=1, HQ=8, h0=1 << 40, d_ht=1 << 40, dh0=1 << 40)
    run = lambda n, **kw: lib.kda_recurrent_bwd_scratch(C.byref(_bwd_args(workspace_bytes=n, **kw)), None, 0, None)      # noqa: E731
    # in passes over the heads: a whole number of q/k heads each; the call takes what holds one (the next check after the scratch is of the alignment)
    row = 16384 * (2 * 2048 + 512 + 32)
    assert [size(passes=n) for n in (0, 1, 2, 3, 32, 99)] == [row * n for n in (32, 32, 16, 11, 1, 1)]
    assert size(passes=4, HQ=4) == (row + 16384 * 1024) * 8 == size(passes=99, HQ=4)
    assert run(size(), d_o=260) == run(size() - 1, d_o=260) == run(row, d_o=260) == -4 and run(row - 1) == -5
    assert run(size(passes=4, HQ=4), HQ=4, d_o=260) == -4 and run(size(passes=4, HQ=4) - 1, HQ=4) == -5
    assert run(size(HQ=1), HQ=1, d_o=260) == -4 and run(size(HQ=1) - 1, HQ=1) == -5
    assert run(1 << 40, K=96) == -2 and run(1 << 40, io_dtype=0) == -3 and run(1 << 40, dq=None) == -1 and run(1 << 40, d_o=260) == -4

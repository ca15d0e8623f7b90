"""CPU: the C-ABI library builds, loads, exports every symbol include/mkda.h declares and agrees with the header on
struct layout; host-side argument checks fail loudly (no compute is launched here)."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from mogankda_b200 import build, _lib
    build.build()
    return _lib.load()


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "mkda.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.findall(r"^\s*(?:int|const char\*)\s+(mkda_\w+)\s*\(", text, flags=re.M)


def test_every_declared_symbol_is_exported(lib):
    names = _declared_functions()
    assert len(names) >= 17
    for n in names:
        assert hasattr(lib, n), n


def test_struct_sizes_match_header(lib):
    from mogankda_b200 import _lib
    n = len(_lib.STRUCT_ORDER)
    sizes = (ctypes.c_int * n)()
    assert lib.mkda_struct_sizes(sizes, n) == n
    for i, name in enumerate(_lib.STRUCT_ORDER):
        assert sizes[i] == ctypes.sizeof(_lib.STRUCTS[name]), name
    assert lib.mkda_abi_version() == 4


# bytes of every parameter struct, by version: a host built against an earlier header of the same version hands over these and no more
LAYOUTS = {4: dict(MkdaLayout=48, MkdaGateFwd=128, MkdaGateBwd=128, MkdaReduce=32, MkdaReduceMulti=96, MkdaL2Norm=32, MkdaIntraFwd=200, MkdaRecurFwd=168,
                   MkdaOutFwd=152, MkdaChainFwd=320, MkdaStepFwd=256, MkdaEpilogueBwd=104, MkdaEpilogueBwdTiles=152, MkdaEpilogueBwdNoAlloc=104,
                   MkdaBwdDh=176, MkdaBwdChunk=256, MkdaQkGrad=128, MkdaCombine=72, MkdaWarmup=80, MkdaSelfTest=40, MkdaSelfTestWait=16)}


def test_struct_layouts_belong_to_the_version(lib):
    """A field more in a struct is read from behind what such a host passes."""
    from mogankda_b200 import _lib
    assert {n: ctypes.sizeof(_lib.STRUCTS[n]) for n in _lib.STRUCT_ORDER} == LAYOUTS[lib.mkda_abi_version()]


def test_null_arguments_are_rejected_without_launch(lib):
    from mogankda_b200 import _lib
    p = _lib.STRUCTS["MkdaIntraFwd"]()
    rc = lib.mkda_intra_fwd(ctypes.byref(p), None)
    assert rc == _lib.MKDA_ERR_ARG
    assert b"intra_fwd" in lib.mkda_last_error()


def test_cpu_tensors_fail_loudly():
    import mogankda_b200 as mk
    q = torch.randn(1, 64, 2, 128)
    with pytest.raises(RuntimeError, match="CUDA"):
        mk.chunk_kda(q, q, q, -torch.rand(1, 64, 2, 128), torch.rand(1, 64, 2))


def test_api_argument_errors():
    import mogankda_b200 as mk
    q = torch.randn(1, 64, 2, 128)
    with pytest.raises(AssertionError):
        mk.chunk_kda(q, q, q, -torch.rand(1, 64, 2), torch.rand(1, 64, 2))          # scalar gate into chunk_kda
    with pytest.raises(AssertionError):
        mk.chunk_gated_delta_rule(q, q, q, -torch.rand(1, 64, 2), torch.rand(1, 64, 2), head_first=True)


def test_product_does_not_import_the_oracle():
    pkg = os.path.join(ROOT, "mogankda_b200")
    for fn in os.listdir(pkg):
        if fn.endswith(".py"):
            assert "oracle" not in open(os.path.join(pkg, fn)).read(), fn


def test_entry_points_reject_misaligned_tensors_without_launching():
    """The kernels use 16-byte vector accesses and bulk copies: a misaligned device address must come back as an error
    code, not as a device fault.  Checked with fake addresses on a machine without a GPU: the check precedes any launch."""
    import ctypes
    from mogankda_b200 import _lib
    lib = _lib.load()
    p = _lib.STRUCTS["MkdaL2Norm"]()
    p.x, p.dtype, p.rows, p.eps, p.rstd = 0x10004, 1, 4, 1e-6, 0x20000
    assert lib.mkda_l2norm_rstd(ctypes.byref(p), None) == -1
    assert b"16-byte aligned" in lib.mkda_last_error()
    q = _lib.STRUCTS["MkdaQkGrad"]()
    q.L.HK, q.L.HV, q.L.NC = 1, 1, 1
    for f in ("dq_v", "dk_v", "q", "k", "dq"):
        setattr(q, f, 0x30000)
    q.dk = 0x30008
    assert lib.mkda_qk_grad_finish(ctypes.byref(q), None) == -1
    assert b"16-byte aligned" in lib.mkda_last_error()


@pytest.mark.parametrize("A", [0, 0x40010, 0x40001])
def test_forward_only_does_not_look_at_A(lib, A):
    """A host may leave the field of mkda_intra_fwd_forward_only as it is; mkda_intra_fwd needs it, aligned.  Without chunks: nothing is launched."""
    from mogankda_b200 import _lib
    p = _lib.STRUCTS["MkdaIntraFwd"]()
    p.L.HK, p.L.HV, p.L.NC, p.A = 1, 1, 0, A
    for f in ("q", "k", "v", "g_c", "beta", "Aqk", "nw", "u", "kbar", "qs", "gl"):
        setattr(p, f, 0x30000)
    assert lib.mkda_intra_fwd_forward_only(ctypes.byref(p), None) == 0
    assert lib.mkda_intra_fwd(ctypes.byref(p), None) == (0 if A and A % 16 == 0 else _lib.MKDA_ERR_ARG)
    p.nw = 0x30001
    assert lib.mkda_intra_fwd_forward_only(ctypes.byref(p), None) == _lib.MKDA_ERR_ARG
    assert lib.mkda_intra_fwd_forward_only(None, None) == _lib.MKDA_ERR_ARG


@pytest.mark.parametrize("scalar", [False, True])
def test_parameter_tensors_of_other_sizes_are_refused(lib, scalar):
    """The kernels take the sizes of A_log, dt_bias and the norm's tensors from v and g; a smaller one would be read, and its gradient written,
    past its end."""
    from mogankda_b200 import _lib
    check, HV = _lib.host().check_params, 4
    v = torch.zeros(1, 8, HV, 128)
    g = v[..., 0] if scalar else v
    A, bias, w = torch.zeros(HV), torch.zeros(HV if scalar else HV * 128), torch.zeros(128)
    for good in ((None,) * 4, (A, bias, w, v), (A.view(1, 1, HV, 1), bias.view(HV, -1), w.view(1, 128), v.view(8, HV * 128))):
        check(v, g, *good)
    other_bias = torch.zeros(HV * 128 if scalar else HV)
    for bad in ((A[:-1], None, None, None), (A.repeat(2), None, None, None), (None, other_bias, None, None), (None, bias[:-1], None, None),
                (None, None, w[:64], None), (None, None, None, v[:, :7]), (None, None, None, v[..., 0])):
        with pytest.raises(AssertionError):
            check(v, g, *bad)


@pytest.mark.parametrize("name", ["_host.so", "libmkda.so"])
def test_modules_share_the_cxx_runtime_of_the_process(lib, name):
    """A second, private copy of the C++ runtime has streams without a locale: formatting a number for an error message crashed the process."""
    import subprocess
    path = os.path.join(ROOT, "mogankda_b200", name)
    needed = subprocess.run(["readelf", "-d", path], capture_output=True, text=True, check=True).stdout
    symbols = subprocess.run(["nm", "-D", "--defined-only", path], capture_output=True, text=True, check=True).stdout
    assert "libstdc++.so.6" in needed
    assert "_ZNSo9_M_insertIlEERSoT_" not in symbols          # std::ostream::_M_insert<long>


def test_a_host_module_of_another_header_is_refused(lib, tmp_path):
    """_host.so has the struct layouts compiled in: against a library with others (here a preloaded mkda_struct_sizes that reports others) the
    import has to fail."""
    import subprocess
    import sys
    src, so = tmp_path / "other.c", tmp_path / "other.so"
    src.write_text("int mkda_struct_sizes(int* out, int n) { for (int i = 0; i < n; ++i) out[i] = 8; return n; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", str(src), "-o", str(so)], check=True)
    code = ("import torch, importlib.util\nspec = importlib.util.spec_from_file_location('mogankda_b200._host', 'mogankda_b200/_host.so')\n"
            "importlib.util.module_from_spec(spec)")
    for preload, ok in (("", True), (str(so), False)):
        run = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, LD_PRELOAD=preload), capture_output=True, text=True)
        assert (run.returncode == 0) == ok, run.stderr
        assert ok or "struct sizes differ" in run.stderr


def test_gate_and_intra_in_one_kernel_refuses_what_it_does_not_take(lib):
    """Without chunks: nothing is launched where the arguments are accepted."""
    from mogankda_b200 import _lib
    g, p = _lib.STRUCTS["MkdaGateFwd"](), _lib.STRUCTS["MkdaIntraFwd"]()
    p.L.HK, p.L.HV, p.L.NC, g.lower_bound, g.mode = 1, 1, 0, -5.0, _lib.MKDA_GATE_EDA
    for s, names in ((p, ("q", "k", "v", "Aqk", "nw", "u", "kbar", "qs", "gl")), (g, ("x", "beta_raw"))):
        for f in names:
            setattr(s, f, 0x30000)
    call = lambda: lib.mkda_gate_intra_fwd(ctypes.byref(g), ctypes.byref(p), None)      # noqa: E731
    assert call() == 0
    for s, f, bad in ((g, "beta_raw", 0), (g, "x", 0x30008), (g, "g_c", 0x30008), (p, "A", 0x30008), (g, "x_dtype", 7), (g, "beta_dtype", -1), (g, "lower_bound", 0.0),
                      (g, "scalar_gate", 1), (p, "nw", 0), (p.L, "HK", 0)):
        good = getattr(s, f)
        setattr(s, f, bad)
        assert call() == _lib.MKDA_ERR_ARG, f
        setattr(s, f, good)
    assert call() == 0
    assert lib.mkda_gate_intra_fwd(None, ctypes.byref(p), None) == _lib.MKDA_ERR_ARG and lib.mkda_gate_intra_fwd(ctypes.byref(g), None, None) == _lib.MKDA_ERR_ARG


def test_finished_chunk_backward_refuses_what_is_left_to_finish(lib):
    """Without chunks: nothing is launched where the arguments are accepted."""
    from mogankda_b200 import _lib
    p = _lib.STRUCTS["MkdaBwdChunk"]()
    p.L.HK, p.L.HV, p.L.NC = 2, 2, 0
    for f in ("q", "k", "v", "g_c", "beta", "A", "h", "dh", "Vd", "dO_t", "dVd_t", "dgp", "dbeta", "dv"):
        setattr(p, f, 0x30000)
    p.dq_v = 0x30001                                       # not looked at
    call = lambda dq=0x30000, dk=0x30000: lib.mkda_bwd_chunk_rows(ctypes.byref(p), None, dq, dk, None)      # noqa: E731
    assert call() == 0
    assert call(dq=0) == call(dk=0) == call(dk=0x30008) == _lib.MKDA_ERR_ARG
    for obj, f, bad in ((p.L, "HV", 4), (p, "q_rstd", 0x30000), (p, "k_rstd", 0x30000), (p, "dv", 0)):
        good = getattr(obj, f)
        setattr(obj, f, bad)
        assert call() == _lib.MKDA_ERR_ARG, f
        setattr(obj, f, good)
    assert lib.mkda_bwd_chunk(ctypes.byref(p), None) == _lib.MKDA_ERR_ARG


def test_reverse_chain_on_rows_refuses_other_rows(lib):
    """Without segments: nothing is launched where the arguments are accepted."""
    from mogankda_b200 import _lib
    p = _lib.STRUCTS["MkdaBwdDh"]()
    p.L.NS, p.do_dtype = 0, _lib.MKDA_BF16
    for f in ("d_o", "kbar", "qs", "gl", "Aqk", "nw"):
        setattr(p, f, 0x30000)
    call = lambda: lib.mkda_bwd_dh_rows(ctypes.byref(p), None, None)                    # noqa: E731
    assert call() == 0                                     # no tiles: no chunk is ragged
    for f, bad in (("d_o", 0), ("d_o", 0x30002), ("do_dtype", _lib.MKDA_F16), ("dO_t", 0x30008), ("nw", 0), ("dh", 0x30010)):
        good = getattr(p, f)
        setattr(p, f, bad)
        assert call() == _lib.MKDA_ERR_ARG, f
        setattr(p, f, good)
    assert lib.mkda_bwd_dh_rows(None, None, None) == _lib.MKDA_ERR_ARG


def test_chunk_backward_on_rows_of_dO_refuses_other_rows(lib):
    """Without chunks: nothing is launched where the arguments are accepted.  dO as rows or as tiles; one of them there has to be."""
    from mogankda_b200 import _lib
    p = _lib.STRUCTS["MkdaBwdChunk"]()
    p.L.HK, p.L.HV, p.L.NC, p.qkv_dtype = 1, 2, 0, _lib.MKDA_BF16
    for f in ("q", "k", "v", "g_c", "beta", "A", "h", "dh", "Vd", "dO_t", "dVd_t", "dq_v", "dk_v", "dgp", "dbeta", "dv"):
        setattr(p, f, 0x30000)
    call = lambda d_o: lib.mkda_bwd_chunk_rows(ctypes.byref(p), d_o, None, None, None)  # noqa: E731
    assert call(0x30000) == call(None) == 0
    assert call(0x30002) == call(0x30008) == _lib.MKDA_ERR_ARG
    for dt in (_lib.MKDA_F16, _lib.MKDA_F32):
        p.qkv_dtype = dt
        assert call(0x30000) == _lib.MKDA_ERR_ARG and call(None) == 0
    p.qkv_dtype, p.dO_t = _lib.MKDA_BF16, None
    assert call(0x30000) == 0 and call(None) == _lib.MKDA_ERR_ARG
    assert lib.mkda_bwd_chunk(ctypes.byref(p), None) == _lib.MKDA_ERR_ARG

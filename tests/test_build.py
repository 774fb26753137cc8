"""The CUDA libraries as files: they build for sm_100a without a GPU and export what the engine
switches at run time (no GPU needed: nothing is launched)."""
import ctypes
import re

import pytest

from vllm_lite_b200.csrc import build, ops


def kernel_libraries():
    for name in build.SOURCES:
        yield name, None
    for name, variants in build.VARIANTS.items():
        for defines in variants:
            yield name, defines


def test_every_kernel_library_builds_and_exports_the_launch_switch():
    """Steps of many tokens are launched without programmatic dependent launch; the switch lives in
    every library (csrc/common.cuh), so a library without it would keep the attribute on."""
    for name, defines in kernel_libraries():
        handle = build.load(name, defines)
        assert isinstance(handle, ctypes.CDLL)
        assert hasattr(handle, "vl_set_pdl"), f"{name} {defines} exports no vl_set_pdl"


def test_the_paired_product_has_no_path_to_dependent_launch():
    """The product on clusters of two blocks stood still on the device now and then when it was started
    as a programmatic dependent.  Its launcher therefore builds its own launch with the cluster attribute
    alone: it neither names the other attribute nor goes through the shared launcher that adds it."""
    import re
    text = (build.CSRC / "gemm_tc5_pair.cu").read_text()
    code = re.sub(r"//[^\n]*", "", text)
    assert "ProgrammaticStreamSerialization" not in code
    assert "vl_launch(" not in code and "vl_pdl_enabled" not in code
    assert re.search(r"cfg\.numAttrs\s*=\s*1\s*;", code) and code.count("numAttrs") == 1
    assert code.count("cudaLaunchKernelEx") == 1
    # the kernels that allocate tensor memory do so behind their wait for the kernels before them
    for name in ("gemm_tc5_pair.cu", "gemm_tc5.cu", "flash_tc5.cu"):
        body = re.sub(r"//[^\n]*", "", (build.CSRC / name).read_text())
        body = body[body.index("__global__"):]
        assert 0 < body.index("pdl_wait();") < body.index("alloc"), name


def test_the_grouped_product_of_paired_blocks_has_no_path_to_dependent_launch():
    import re
    code = re.sub(r"//[^\n]*", "", (build.CSRC / "gemm_tc5_grouped.cu").read_text())
    assert "ProgrammaticStreamSerialization" not in code and "vl_launch(" not in code and "vl_pdl_enabled" not in code
    assert re.search(r"cfg\.numAttrs\s*=\s*1\s*;", code) and code.count("numAttrs") == 1 and code.count("cudaLaunchKernelEx") == 1
    body = code[code.index("__global__"):]
    assert 0 < body.index("pdl_wait();") < body.index("alloc_pair")


# A wait is given up by each lane at its own time.  Where the lanes then meet again (a warp's barrier, a load of tensor memory), one that left
# by itself would let the others wait for good: whoever breaks off a loop over a wait does so by the vote of the warp.
@pytest.mark.parametrize("name", ["gemm_tc5", "gemm_tc5_pair", "gemm_tc5_grouped", "gemm_few", "gemm_batched", "flash_tc5", "gemm_bf16"])
def test_no_lane_leaves_a_loop_by_itself_when_a_wait_runs_out(name):
    code = re.sub(r"//[^\n]*", "", (build.CSRC / f"{name}.cu").read_text())
    assert "wait" in code and not re.search(r"if\s*\(\s*!\s*(tc5::)?mbar_wait_bounded", code)
    assert "__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity))" in (build.CSRC / "tc5.cuh").read_text()


def test_capped_scores_are_scaled_and_then_capped():
    """The two-at-a-time form of `shape_score` keeps its order: the score times the scale, that times 2 / cap.  The factors' own product first rounds
    elsewhere, which moves last bits of every capped layer."""
    code = re.sub(r"//[^\n]*", "", (build.CSRC / "flash_tc5.cu").read_text())
    assert "scale_log2 * toc" not in code and "toc * scale_log2" not in code
    assert "k2 = pair(scale_log2, scale_log2), t2 = pair(toc, toc)" in code and code.count("k2, zero2), t2, zero2)") == 1


def test_the_weight_streams_consumers_leave_together():
    """Between two tiles the four consumer warps meet at barriers that count 128 threads, and their lanes behind every stage: one that left
    alone behind a wait that ran out would keep the others there.  So a wait notes for the block that it gave up, no loop over stages is left, and
    all ask between the tile's two barriers."""
    code = re.sub(r"//[^\n]*", "", (build.CSRC / "gemm_bf16.cu").read_text())
    stages = code[code.index("auto multiply = "):code.index("for (int n0 = r0; n0 < r1; n0 += GS_ROWS) {\n#pragma unroll")]
    assert "mbar_wait_or_note(" in stages and "return" not in stages
    tile = code[code.index("for (int n0 = r0; n0 < r1; n0 += GS_ROWS) {\n#pragma unroll"):]
    first = tile.index("consumer_barrier();")
    asked, second, left = tile.index("const bool ok = !s_gave_up;"), tile.index("consumer_barrier();", first + 1), tile.index("if (!ok) {")
    assert first < asked < second < left and tile[:left].count("break;") == 1            # (the last of an odd number of stages)


def test_the_engine_is_imported_without_a_compiler(tmp_path):
    """An import builds nothing: without a compiler on the path and without built files the package, its engine and the checks of `ops`
    are there; only a launch needs more."""
    import os
    import shutil
    import subprocess
    import sys
    root = build.CSRC.parent.parent
    for package in ("vllm_lite_b200", "vllm-lite_b200"):
        shutil.copytree(root / package, tmp_path / package, ignore=shutil.ignore_patterns("_build", "__pycache__"))
    code = """
import torch
import vllm_lite_b200.engine
from vllm_lite_b200.csrc import ops
try:
    ops.cast(torch.zeros(4), torch.zeros(4))
except ops.KernelError as e:
    print("refused:", e)
"""
    hidden = {k: v for k, v in os.environ.items() if k not in ("CXX", "NVCC", "CUDA_HOME", "PYTHONPATH")}
    hidden.update(PATH=str(tmp_path), TMPDIR=str(tmp_path))
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=tmp_path, env=hidden)
    assert run.returncode == 0 and "CUDA tensor" in run.stdout, run.stderr
    assert not list(tmp_path.rglob("*.so"))


def test_dependent_launch_is_off_until_switched_on():
    assert ops._pdl is False or ops._pdl_libs            # the module's default; a test before may have stepped
    for name, defines in kernel_libraries():
        handle = build.load(name, defines)
        if (name, build._variant(defines)) not in ops._pdl_libs:
            assert handle.vl_get_pdl() == 0, name


def test_digest_covers_every_header():
    """A library is rebuilt when any header beside the sources changes, plain C headers included."""
    import hashlib
    before = build._digest("attention")
    h = build.CSRC / "zz_probe_header.h"
    try:
        h.write_text("// probe\n")
        assert build._digest("attention") != before
    finally:
        h.unlink()
    assert build._digest("attention") == before


def test_set_pdl_reaches_the_libraries_that_are_loaded():
    calls = []
    saved, saved_flag = dict(ops._pdl_libs), ops._pdl
    try:
        ops._pdl_libs.clear()
        ops._pdl_libs[("fake", "")] = calls.append
        ops.set_pdl(not saved_flag)
        ops.set_pdl(not saved_flag)              # no change: nothing is called again
        ops.set_pdl(saved_flag)
        assert calls == [int(not saved_flag), int(saved_flag)]
    finally:
        ops._pdl_libs.clear()
        ops._pdl_libs.update(saved)
        ops._pdl = saved_flag


def test_ctypes_signatures_match_the_c_declarations():
    """The engine calls its libraries through ctypes, where nothing checks an argument list: a float
    passed where the C side reads an int goes wrong silently.  So the declarations are read from the
    sources and compared, kind by kind (pointer, int, 64-bit int, float), with what ops.py binds."""
    import re
    declared = {}
    for path in build.CSRC.glob("*.cu"):
        for m in re.finditer(r'extern "C" int (\w+)\(([^)]*)\)\s*\{', path.read_text(), re.S):
            declared[(path.stem, m.group(1))] = [a.strip() for a in m.group(2).replace("\n", " ").split(",") if a.strip()]

    def c_kind(arg):
        if "*" in arg:
            return "pointer"
        type_words = " ".join(arg.split()[:-1])
        if "float" in type_words:
            return "float"
        if "long long" in type_words or "size_t" in type_words or "int64" in type_words:
            return "int64"
        return "int"

    py_kind = {ctypes.c_void_p: "pointer", ctypes.c_float: "float", ctypes.c_int: "int",
               ctypes.c_longlong: "int64", ctypes.c_size_t: "int64"}
    assert ops._SIGNATURES
    for key, bound in ops._SIGNATURES.items():
        assert key in declared, f"{key} is bound but not declared extern C in its source"
        assert [c_kind(a) for a in declared[key]] == [py_kind[t] for t in bound], key


def test_host_core_bindings_match_the_c_declarations():
    """The same check for the C++ core of cache manager and scheduler (cache/native.py)."""
    import re
    from ctypes import c_int, c_longlong
    from vllm_lite_b200.cache import native
    lib = native._core()
    text = (build.CSRC / "host" / "cache_core.cpp").read_text()
    found = 0
    for m in re.finditer(r"^\s*([\w \*]+?)\s*\b(v[cs]_\w+)\(([^)]*)\)\s*\{", text, re.S | re.M):
        ret, name, args = m.group(1).strip(), m.group(2), [a.strip() for a in m.group(3).replace("\n", " ").split(",") if a.strip()]
        fn = getattr(lib, name)
        assert fn.argtypes is not None, f"{name} is exported but not bound"

        def c_kind(text_type):
            if "*" in text_type:
                return "pointer"
            return "int64" if "long long" in text_type else "int"

        def py_kind(t):
            return {c_int: "int", c_longlong: "int64"}.get(t, "pointer")

        assert [c_kind(" ".join(a.split()[:-1]) if "*" not in a else a) for a in args] == [py_kind(t) for t in fn.argtypes], name
        want = "void" if ret == "void" else c_kind(ret)
        assert want == ("void" if fn.restype is None else py_kind(fn.restype)), name
        found += 1
    assert found >= 19


def test_entry_points_are_called_as_ctypes_calls_them(tmp_path):
    """The extension module hands whole numbers and floats to a C function by the calling convention's own rules; ctypes is the
    reference, for argument lists longer than the registers and with floats anywhere between."""
    import random
    import subprocess
    import pytest
    bind = build.load_ext("bind")
    kinds = {"p": ("const void*", ctypes.c_void_p), "i": ("int", ctypes.c_int), "l": ("long long", ctypes.c_longlong), "f": ("float", ctypes.c_float)}
    rng = random.Random(5)
    sigs = ["p", "f", "ffffffff", "i" * 30, "pifl" * 8] + ["".join(rng.choice("ppiilf" if k < 8 else "ppiil") for k in range(rng.randint(1, 38)))
                                                           for _ in range(12)]
    sigs = [s for s in sigs if s.count("f") <= 8]
    body = ""
    for n, s in enumerate(sigs):
        args = ", ".join(f"{kinds[k][0]} a{i}" for i, k in enumerate(s))
        terms = " ".join(f"s = s * 31 + (long long)({'a%d * 8' % i if k == 'f' else '(long long)a%d' % i});" for i, k in enumerate(s))
        body += f'extern "C" int f{n}({args}) {{ unsigned long long s = 7; {terms} return (int)(s % 1000003); }}\n'
    (tmp_path / "f.cpp").write_text(body)
    subprocess.run([build.find_cxx(), "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "f.so"), str(tmp_path / "f.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "f.so"))
    for n, s in enumerate(sigs):
        fn = getattr(lib, f"f{n}")
        fn.argtypes, fn.restype = [kinds[k][1] for k in s], ctypes.c_int
        entry = bind.Entry(ctypes.cast(fn, ctypes.c_void_p).value, s)
        for _ in range(3):
            args = [{"p": rng.choice([None, rng.randrange(1 << 47)]), "i": rng.randint(-(1 << 31), (1 << 31) - 1),
                     "l": rng.randint(-(1 << 62), 1 << 62), "f": rng.randint(-4000, 4000) / 8}[k] for k in s]
            assert entry(*args) == fn(*args), s
        with pytest.raises(TypeError):
            entry(*args, 0)
    with pytest.raises(TypeError):
        bind.Entry(ctypes.cast(lib.f0, ctypes.c_void_p).value, "i")("text")
    for bad in ("x", "f" * 9, "i" * 41):
        with pytest.raises(ValueError):
            bind.Entry(1, bad)


def test_every_kernel_reports_a_wait_that_ran_out_under_its_own_name():
    from vllm_lite_b200.engine.runner import _DEVICE_ERRORS
    bits = {m.group(1): int(m.group(2), 16) for m in re.finditer(r"#define (VL_DEV_IN_\w+) (0x[0-9a-f]+)u", (build.CSRC / "common.cuh").read_text())}
    roles = [1 << (16 + i) for i in range(4)]
    assert len(set(bits.values())) == len(bits) and all(b & (b - 1) == 0 and b not in roles and b in _DEVICE_ERRORS for b in bits.values())
    assert len(set(_DEVICE_ERRORS.values())) == len(_DEVICE_ERRORS)
    users = {}
    for path in build.CSRC.glob("*.cu"):
        for name in set(re.findall(r"VL_DEV_IN_\w+", path.read_text())):
            users.setdefault(name, []).append(path.stem)
    assert set(users) == set(bits) and all(len(files) == 1 for files in users.values()), users


def test_the_library_product_is_torchs_own_in_all_its_forms():
    """`ops.mm` goes through the dispatcher with all of its keys: a gradient is refused, modes and tensor types of somebody's own are
    asked, warnings and errors are torch's (the product itself runs on the CPU here)."""
    import torch
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Functions(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func.__name__)
            return func(*args, **(kwargs or {}))

    class Calls(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func.__name__)
            return func(*args, **(kwargs or {}))

    class Own(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(func.__name__)
            return super().__torch_function__(func, types, args, kwargs or {})

    seen = []
    a, w = torch.randn(5, 8), torch.randn(3, 8)
    out, want = torch.empty(5, 3), a @ w.t()
    assert ops.mm(a, w, out) is out and torch.equal(out, torch.mm(a, w.t()))
    for bad in ((a.clone().requires_grad_(), w, out), (a, torch.nn.Parameter(w), out)):
        for product in (ops.mm, ops._torch_mm):
            with pytest.raises(RuntimeError, match="automatic differentiation"):
                product(*bad)
        with torch.no_grad():
            assert torch.equal(ops.mm(*bad), want)
    for mode in (Functions, Calls):
        with mode():
            ops.mm(a, w, out)
        assert any(name.startswith("mm") for name in seen), mode
        seen.clear()
    ops.mm(a.as_subclass(Own), w, out)
    assert "mm" in seen
    with pytest.raises(RuntimeError, match="shapes cannot be multiplied"):
        ops.mm(a, torch.randn(3, 7), out)
    with pytest.warns(UserWarning, match="resized"):
        ops.mm(a, w, torch.empty(1, 3))
    with pytest.raises(TypeError):
        ops.mm(a, w, None)

"""CPU-side checks of the boundary: the library loads, exports every symbol the header
declares, and rejects bad arguments before touching a device."""
import ctypes
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HEADER = ROOT / "include" / "fss_b200.h"


def declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(fss_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from fast_sequential_scan_b200 import _lib
    L = _lib.lib()
    names = declared_functions()
    assert len(names) >= 15
    for name in names:
        assert hasattr(L, name), f"{name} declared in include/fss_b200.h but not exported"
    assert sorted(_lib.SIGNATURES) == names, "ctypes table and header disagree"
    assert L.fss_abi_version() == 1


def test_struct_layouts_match_the_header():
    from fast_sequential_scan_b200 import _lib
    assert ctypes.sizeof(_lib.View) == 24
    assert ctypes.sizeof(_lib.ScanCtx) == 48
    assert ctypes.sizeof(_lib.ForwardState) == 40 and ctypes.sizeof(_lib.BackwardState) == 40


def test_carry_source_and_flag_constants_match_the_header():
    """Field order of fss_carry_source and the values of the FSS_FLAG_* / FSS_ALGO_* constants, read from the header text."""
    from fast_sequential_scan_b200 import _lib
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    body = re.search(r"typedef struct fss_carry_source \{(.*?)\} fss_carry_source;", text, flags=re.S).group(1)
    fields = []
    for decl in body.split(";"):
        decl = decl.strip()
        if decl:
            fields += [re.sub(r"[^A-Za-z0-9_]", "", part.split()[-1]) for part in decl.split(",")]
    assert fields == [name for name, _ in _lib.CarrySource._fields_]
    assert ctypes.sizeof(_lib.CarrySource) == 72
    defines = dict(re.findall(r"#define (FSS_(?:FLAG|ALGO)_[A-Z_]+) (0x[0-9a-fA-F]+|\d+)", text))
    assert len(defines) >= 7
    for name, value in defines.items():
        assert getattr(_lib, name[4:]) == int(value, 0), f"{name}: header {value}, ctypes {getattr(_lib, name[4:])}"


def test_error_strings_and_argument_checks_need_no_device():
    from fast_sequential_scan_b200 import _lib
    L = _lib.lib()
    assert L.fss_strerror(0) == b"ok"
    for code in range(-12, 0):
        assert L.fss_strerror(code) != b"unknown error code"
    v = _lib.View(0, 0, 0)
    ctx = _lib.ScanCtx(ctypes.sizeof(_lib.ScanCtx), -1, None, None, 0, None, 0, 0)
    call = lambda c, B, T, D, *views: L.fss_scan_forward_half(ctypes.byref(c), B, T, D, *[ctypes.byref(x) for x in views])
    assert call(ctx, 2, 4, 8, v, v, v) == -1                       # NULL tensor
    assert call(ctx, -1, 4, 8, v, v, v) == -2                      # negative extent
    assert call(ctx, 0, 4, 8, v, v, v) == 0                        # empty problem: nothing to do
    bad = _lib.ScanCtx(8, -1, None, None, 0, None, 0, 0)
    assert call(bad, 2, 4, 8, v, v, v) == -10                      # struct size skew
    ctx.algo = 9
    assert call(ctx, 2, 4, 8, v, v, v) == -7
    ctx.algo = 0
    buf = (ctypes.c_uint16 * 64)()
    p = _lib.View(ctypes.addressof(buf), 32, 4)                    # row stride 4 < D = 8
    assert call(ctx, 2, 4, 8, p, p, p) == -2
    ok = [_lib.View(ctypes.addressof(buf) + 128 * k, 32, 8) for k in range(3)]
    assert call(ctx, 2, 4, 8, *ok) == -4                           # no workspace
    assert call(ctx, 2, 4, 8, ok[0], ok[1], ok[0]) == -12          # h starts where alpha starts
    assert call(ctx, 2, 4, 8, ok[0], ok[1], ok[1]) == -12          # ... or where beta starts
    # the chunked kernels run on a linear grid of (channel blocks x chunks x batch) CTAs; a problem
    # whose grid would not fit 31 bits is refused instead of being launched with a truncated grid
    T, D = 1 << 34, 1 << 14
    huge = [_lib.View(ctypes.addressof(buf) + 128 * k, T * D, D) for k in range(3)]
    ctx.algo = _lib.ALGO_CHUNKED
    assert call(ctx, 64, T, D, *huge) == -2
    ctx.algo = 0
    wide = _lib.View(ctypes.addressof(buf), 1 << 62, 8)            # batch stride whose extent overflows
    assert call(ctx, 16, 4, 8, wide, ok[1], ok[2]) == -2
    assert L.fss_workspace_bytes(8, 2048, 1024, 0) > 256
    assert L.fss_workspace_bytes(0, 0, 0, 0) >= 256
    assert L.fss_block_rows(0, 1, 65536, 4096, 1) >= 1


# dtype, B, T, D of single-pass problems: both sides of 64 MiB a tensor and 384 columns of 64 bytes, wide ones, short ones
TILE_SHAPES = [("f32", 4, 4096, 2048), ("f32", 4, 2048, 1024), ("f32", 2, 8192, 2560), ("bf16", 16, 2048, 1024), ("bf16", 4, 4096, 2048),
               ("bf16", 16, 4096, 2560), ("f32", 16, 4096, 2560), ("bf16", 2, 300, 768), ("bf16", 1, 40, 512)]


def _tile_rows(forced):
    """Rows per tile of forward, reversed forward and backward launches, in a process of its own (the switch is read once)."""
    code = ("import ctypes, sys; L = ctypes.CDLL(sys.argv[1]); L.fss_tile_rows.restype = ctypes.c_int64\n"
            "for a in sys.argv[2:]:\n"
            "    dt, B, T, D = a.split(',')\n"
            "    print(*[L.fss_tile_rows(int(dt == 'f32'), bwd, *map(ctypes.c_int64, (int(B), int(T), int(D))), flags)"
            " for bwd, flags in ((0, 0), (0, 8), (1, 0), (1, 8))])")
    from fast_sequential_scan_b200 import _lib
    env = {k: v for k, v in os.environ.items() if k not in ("FSS_B200_SPLIT", "FSS_B200_TAIL", "FSS_B200_TICKETS")}
    if forced:
        env["FSS_B200_SPLIT"] = str(forced)
    out = subprocess.run([sys.executable, "-c", code, str(_lib.LIB_PATH), *[",".join(map(str, c)) for c in TILE_SHAPES]],
                         capture_output=True, text=True, check=True, env=env).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


@pytest.mark.parametrize("forced", [1, 2, 4])
def test_forced_tile_shape_holds_for_every_problem(forced):
    assert _tile_rows(forced) == [(64 * forced,) * 4] * len(TILE_SHAPES)


def test_tile_shapes_chosen_by_default():
    rows = _tile_rows(None)
    assert rows == [(128, 128, 256, 256), (256,) * 4, (256,) * 4, (128,) * 4, (256,) * 4, (64,) * 4, (64,) * 4, (128,) * 4, (64,) * 4]


def test_package_has_no_fallback_when_library_is_missing(monkeypatch, tmp_path):
    from fast_sequential_scan_b200 import _lib
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setenv("FSS_B200_LIB", str(tmp_path / "nope.so"))
    with pytest.raises(ImportError):
        _lib.lib()
    monkeypatch.delenv("FSS_B200_LIB")
    monkeypatch.setattr(_lib, "_lib", None)
    _lib.lib()


def test_product_never_imports_the_oracle():
    pkg = ROOT / "fast_sequential_scan_b200"
    for path in list(pkg.rglob("*.py")) + list(pkg.rglob("*.cu*")):
        text = path.read_text()
        assert "oracle" not in text.replace("# oracle", ""), f"{path} mentions the oracle"


def test_python_surface_mirrors_the_reference_names():
    import fast_sequential_scan_b200 as pkg
    from fast_sequential_scan_b200 import scan_cuda, sequential_scan_cuda as native
    assert callable(pkg.scan_cu) and callable(pkg.scan_cu_single)
    for name in ("SequentialScan", "SequentialScanSingle", "scan", "scan_single"):
        assert hasattr(scan_cuda, name)
    for name in ("scan_forward", "scan_backward", "scan_forward_half", "scan_backward_half"):
        assert callable(getattr(native, name))


def test_backward_mode_switch_validates_its_argument():
    from fast_sequential_scan_b200 import scan_cuda
    assert scan_cuda.BACKWARD_MODES == ("saved", "inplace", "recompute")
    previous = scan_cuda.set_backward_mode("recompute")
    try:
        assert previous == "saved" and scan_cuda._resolve(None) == "recompute"
        assert scan_cuda._resolve("inplace") == "inplace"
        with pytest.raises(ValueError):
            scan_cuda.set_backward_mode("in-place")
        with pytest.raises(ValueError):
            scan_cuda._resolve("keep")
    finally:
        scan_cuda.set_backward_mode(previous)


def test_reference_arm_of_the_bench_prints_the_contract_line():
    """`bench.py --impl reference` runs on host cores only; one JSON line with the agreed keys."""
    import json
    import subprocess
    import sys
    root = Path(__file__).resolve().parent.parent
    out = subprocess.run([sys.executable, str(root / "bench.py"), "--impl", "reference", "--workload", "c1",
                          "--steps", "2", "--warmup", "1"], capture_output=True, text=True, timeout=300, cwd=root)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["higher_is_better"] is True and line["value"] > 0
    for key in ("metric", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "config", "cpu_baseline", "e2e"):
        assert key in line
    assert line["cpu_baseline"]["kind"] in ("reference", "port") and line["cpu_baseline"]["cores"] >= 1
    assert line["e2e"]["h2d_bytes_per_step"] == 0 and line["e2e"]["d2h_bytes_per_step"] == 0


def test_kernels_that_start_early_do_not_take_their_predecessors_data_for_constant():
    """The gated scans and the kernels that make their tables are placed while the kernel before them runs.  A load that
    is only defined for data that stay constant for the kernel's life (``__ldg``, or what the compiler makes of a
    ``const __restrict__`` pointer) must not read what that kernel writes: the tables, lambda."""
    csrc = ROOT / "fast_sequential_scan_b200" / "csrc"
    lookback, gates = (re.sub(r"//[^\n]*", "", (csrc / n).read_text()) for n in ("fss_lookback.cuh", "fss_gates.cuh"))
    assert "__ldg" not in lookback
    for kernel in ("prescale", "backward_tables"):
        arguments = re.search(rf"__global__ void {kernel}\((.*?)\) \{{", gates, flags=re.S).group(1)
        assert "__restrict__" not in arguments, kernel


@pytest.mark.parametrize("content", [None, b"not a shared object"])
def test_import_without_the_cpp_autograd_functions(tmp_path, content):
    """The Python classes serve every call by themselves: a missing ``_fss_torch`` file, or one that does not load, is a
    warning.  A file that was built for another torch is not looked at."""
    import shutil
    import subprocess
    import sys
    package = ROOT / "fast_sequential_scan_b200"
    copy = tmp_path / package.name
    shutil.copytree(package, copy, ignore=shutil.ignore_patterns("*.so", "csrc", "__pycache__"))
    (copy / "libfss_b200.so").symlink_to(package / "libfss_b200.so")
    (copy / "_fss_torch.so").write_bytes(b"of another torch")
    if content is not None:
        from fast_sequential_scan_b200.build import torch_lib
        (copy / torch_lib().name).write_bytes(content)
    code = ("import warnings, torch\n"
            "with warnings.catch_warnings(record=True) as seen:\n"
            "    warnings.simplefilter('always')\n"
            "    import fast_sequential_scan_b200 as pkg\n"
            "    from fast_sequential_scan_b200 import scan_cuda\n"
            "assert [w for w in seen if '_fss_torch' in str(w.message)], seen\n"
            "assert not scan_cuda._ordinary_call(torch.ones(1, 2, 3))\n"
            "try: pkg.scan_cu(torch.ones(1, 2, 3).bfloat16(), torch.ones(1, 2, 3).bfloat16())\n"
            "except RuntimeError as e: assert 'CUDA tensor' in str(e)\n"
            "else: raise AssertionError('no refusal')\n"
            "print('imported from', pkg.__file__)\n")
    out = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and str(tmp_path) in out.stdout, out.stdout + out.stderr


def test_the_cpp_autograd_functions_load_here():
    from fast_sequential_scan_b200 import scan_cuda
    assert scan_cuda._fss_torch is not None

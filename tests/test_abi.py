"""The C-ABI library: it loads, exports every entry point include/nimbus_cuda.h
declares, its argument blocks have the layout the ctypes binding assumes, and
it refuses to run without an sm_100 device (there is no CPU fallback).  No
compute call is made here."""
import ctypes
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest

from nimbus_b200 import cuda

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "include" / "nimbus_cuda.h"


def declared_functions():
    text = HEADER.read_text()
    return sorted(set(re.findall(r"^\s*(?:nimbus_status|void\*?|const char\*|int|uint64_t|size_t)\s+(nimbus_\w+)\(",
                                 text, re.M)))


def test_header_declares_what_binding_expects():
    assert set(declared_functions()) == set(cuda.EXPORTED_SYMBOLS)


def test_library_exports_every_declared_symbol():
    lib = cuda.load_library()
    for name in declared_functions():
        assert hasattr(lib, name), name
    assert lib.nimbus_cuda_abi_version() == 1


def _c_layout(struct_name, fields, tmp_path):
    src = tmp_path / "layout.c"
    lines = ['#include <stdio.h>', '#include <stddef.h>', f'#include "{HEADER}"', "int main(void){",
             f'printf("%zu\\n", sizeof({struct_name}));']
    lines += [f'printf("%zu\\n", offsetof({struct_name}, {f}));' for f in fields]
    lines.append("return 0;}")
    src.write_text("\n".join(lines))
    exe = tmp_path / "layout"
    subprocess.run(["gcc", str(src), "-o", str(exe)], check=True)
    vals = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    return vals[0], vals[1:]


@pytest.mark.parametrize("struct_name,cls", [
    ("nimbus_acoustic_fused_args", cuda.AcousticFusedArgs),
    ("nimbus_acoustic_batched_args", cuda.AcousticBatchedArgs),
    ("nimbus_scalar_transport_args", cuda.ScalarTransportArgs),
    ("nimbus_slow_args", cuda.SlowArgs),
    ("nimbus_kessler_args", cuda.KesslerArgs),
    ("nimbus_eos_args", cuda.EosArgs),
    ("nimbus_sound_speed_args", cuda.SoundSpeedArgs),
    ("nimbus_slow_apply_args", cuda.SlowApplyArgs),
    ("nimbus_kessler_pointwise_args", cuda.KesslerPointwiseArgs),
    ("nimbus_kessler_sedimentation_args", cuda.KesslerSedimentationArgs),
    ("nimbus_cgrid_slow_tendencies_args", cuda.CgridSlowTendenciesArgs),
    ("nimbus_device_info", cuda.DeviceInfo),
    ("nimbus_boundary_args", cuda.BoundaryArgs),
    ("nimbus_state_relaxation_args", cuda.StateRelaxationArgs),
    ("nimbus_cell_centre_args", cuda.CellCentreArgs),
    ("nimbus_smagorinsky_args", cuda.SmagorinskyArgs),
    ("nimbus_sgs_apply_args", cuda.SgsApplyArgs),
    ("nimbus_sgs_stability", cuda.SgsStability),
    ("nimbus_sgs_step_args", cuda.SgsStepArgs),
    ("nimbus_history_args", cuda.HistoryArgs),
    ("nimbus_member_desc", cuda.MemberDesc),
    ("nimbus_engine_tuning", cuda.EngineTuning),
    ("nimbus_member_state", cuda.MemberState),
])
def test_argument_block_layout_matches_header(struct_name, cls, tmp_path):
    fields = [f for f, _ in cls._fields_]
    size, offsets = _c_layout(struct_name, fields, tmp_path)
    assert size == ctypes.sizeof(cls)
    assert offsets == [getattr(cls, f).offset for f in fields]


def test_reference_backend_adapter_exports():
    """The ComputeBackend adapter loads and exposes its factory hooks (no
    backend is created here)."""
    path = ROOT / "nimbus_b200" / "lib" / "libnimbus_reference_backend.so"
    if not path.exists():
        pytest.skip("adapter not built (no reference headers)")
    lib = ctypes.CDLL(str(path))
    assert hasattr(lib, "nimbus_cuda_create_compute_backend")
    assert hasattr(lib, "nimbus_cuda_destroy_compute_backend")


def test_no_device_is_an_error_not_a_fallback():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    with pytest.raises(cuda.NimbusCudaError) as exc:
        cuda.Context(0)
    assert exc.value.status == 6  # NIMBUS_ERR_NO_DEVICE
    backend = cuda.CudaComputeBackend()
    assert backend.initialize() is False and "NO_DEVICE" in backend.last_error


def test_argument_blocks_keep_their_arrays_alive():
    """Argument blocks hold raw pointers; the binding must keep every array
    they point at alive even when the caller passed temporaries."""
    import gc

    import numpy as np

    shape = (6, 5, 4)

    def tmp():
        return np.random.default_rng(0).random(shape).astype(np.float32)

    a = cuda.transport_args([tmp(), tmp()], [tmp(), tmp()], [0, 1], tmp(), tmp(), tmp(), tmp(), tmp(), 1.0,
                            (1.0, 1.0, 1.0))
    st = {k: tmp() for k in ("u", "v", "w", "rho", "p", "theta")}
    b = cuda.batched_args(st, np.ones(4), np.ones(4), 0.1, 2, (1.0, 1.0, 1.0), (1, 1, 1, 1, 1, 0), tmp(), tmp(),
                          tmp(), 0.5, None, np.zeros(2 * 11 * 4, np.float32), tmp())
    del st
    gc.collect()

    def kept_addresses(block):
        out = set()
        for item in block._keep:
            items = item.values() if isinstance(item, dict) else (item if isinstance(item, list) else [item])
            for arr in items:
                if isinstance(arr, np.ndarray):
                    out.add(arr.ctypes.data)
        return out

    for block, names in ((a, ("rho_end", "rho_begin", "mass_flux_x", "mass_flux_y", "mass_flux_z")),
                         (b, ("u", "rho", "theta", "rho0_base", "mass_flux_z", "wave_history_output",
                              "density_begin"))):
        kept = kept_addresses(block)
        for name in names:
            addr = ctypes.cast(getattr(block, name), ctypes.c_void_p).value
            assert addr in kept, name
    for i in range(2):
        assert ctypes.cast(a.q_in[i], ctypes.c_void_p).value in kept_addresses(a)


def test_engine_calls_make_their_device_current_before_they_enqueue():
    """CUDA refuses a launch or an allocation on a stream of another device
    than the calling thread's: every engine entry point that enqueues any makes
    the engine's device current first (itself or in prepare_image)."""
    text = (ROOT / "nimbus_b200" / "csrc" / "engine.cu").read_text()
    text = re.sub(r"//[^\n]*", "", text[text.index('extern "C" {'):])
    starts = [m for m in re.finditer(r"^[\w ]+\*? ?(nimbus_cuda_engine_\w+)\([^;{]*\)\s*\{", text, re.M)]
    enqueues = re.compile(r"<<<|\bmove_state\(|\blaunch_\w+\(|\benqueue\w*\(|cudaMalloc\w*\(|cudaGraphLaunch\(")
    current = re.compile(r"cudaSetDevice\(|\bprepare_image\(")
    checked = []
    for m, following in zip(starts, starts[1:] + [None]):
        body = text[m.end():following.start() if following else len(text)]
        first = enqueues.search(body)
        if first:
            device = current.search(body)
            assert device and device.start() < first.start(), m.group(1)
            checked.append(m.group(1))
    assert {"nimbus_cuda_engine_read_async", "nimbus_cuda_engine_write_async", "nimbus_cuda_engine_admit",
            "nimbus_cuda_engine_step"} <= set(checked)


def test_a_member_takes_no_more_memory_than_its_unpadded_cells():
    """Columns are padded to a multiple of four levels; a member's footprint
    stays within the 44 values a cell (and the tables and alignment) that one
    without padding takes when no buffer serves twice."""
    lib = cuda.load_library()
    for nz in range(14, 81):
        base = {k: np.ones(nz) for k in ("rho0", "p0", "qv0", "u0", "v0")}
        desc = cuda.member_desc((23, 19, nz), (500.0, 500.0, 300.0), 3.0, 4, (1, 1, 1, 1, 1, 0), base)
        cells, faces = 23 * 19 * nz, 2 * (23 + 19) * nz
        bound = 4 * (44 * cells + faces) + 64 * nz + 26 * 256
        assert 0 < lib.nimbus_cuda_engine_member_bytes(ctypes.byref(desc)) <= bound, nz

"""The four-cells-per-thread passes of the member engine and of the
per-operation acoustic loop where their groups end: columns of every length
modulo four (the engine pads them), the smallest grids, lateral rows next to
the walls, every boundary set, and grids on both sides of the size from which
the groups are launched; against the restatement of the reference, bit for
bit in reference precision, and the FP32 engine against the FP32
per-operation path."""
import ctypes

import numpy as np
import pytest

import oracle
from nimbus_b200 import cuda
from nimbus_b200.initial import Case, cloudy_state, perturbed_state
from nimbus_b200.run import EngineRun, ResidentRun

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not oracle.restatement_available(), reason="restatement oracle not built")]

OPEN, CHANNEL, WALLS = (1, 1, 1, 1, 1, 0), (0, 0, 0, 0, 0, 2), (2, 3, 4, 3, 0, 1)
FIELDS = ("u", "v", "w", "rho", "p", "theta", "qv", "qc", "qr")
QUAD_CELLS = 4 * 128 * 4 * 148  # stored cells from which the acoustic passes take groups of four
# (nx, ny, nz): every nz mod 4 (2 and 3 are the shortest columns), the
# narrowest members, 128-cell tiles that end inside a column.
GRIDS = [(4, 4, 2), (5, 4, 3), (4, 7, 5), (9, 8, 6), (8, 11, 9), (13, 6, 12), (17, 19, 23), (12, 31, 41)]


def _same(got, want, what):
    bad = np.flatnonzero(got.view(np.uint32).ravel() != want.view(np.uint32).ravel())
    assert bad.size == 0, f"{what}: {bad.size} of {got.size} values differ, first at {bad[:1]}"


@pytest.fixture(scope="module")
def ctx():
    c = cuda.Context(0)
    yield c
    c.set_precision(cuda.PRECISION_REFERENCE)


def _case(shape, bc, m):
    nx, ny, nz = shape
    return Case(nx, ny, nz, 900.0, 850.0, 20000.0 / max(nz, 20), 2.0, bc=bc, seed=11, member=m)


@pytest.mark.parametrize("large", [None, (88, 87, 41)], ids=["one-cell", "quads"])
@pytest.mark.parametrize("bc", [OPEN, CHANNEL, WALLS], ids=["open", "channel", "walls"])
def test_engine_step_on_every_column_length(ctx, bc, large):
    """Lanes below the size from which the acoustic passes take four cells a
    thread, and one lane that a large member takes above it: the lane's total
    decides, so the small members' columns go through the groups too, in every
    substep (the large member has the most)."""
    run = EngineRun(ctx, precision=cuda.PRECISION_REFERENCE, lanes=1 if large else None)
    cpu = oracle.Restatement("f32")
    members = []
    for m, shape in enumerate(GRIDS + ([large] if large else [])):
        case = _case(shape, bc, m)
        st, base = cloudy_state(case, seed=20 + m)
        n = 6 if shape == large else 3 + m % 3
        members.append((run.admit(case, st, base, coriolis_f=1e-4, n_substeps=n), case, st, base, n))
    stored = sum(c.nx * c.ny * (-(-c.nz // 4) * 4) for _, c, _, _, _ in members)
    assert (stored >= QUAD_CELLS) == bool(large)
    run.step(2)
    for mid, case, st, base, n in members:
        want = {k: v.copy() for k, v in st.items()}
        for _ in range(2):
            cpu.large_step(want, base, (case.dx, case.dy, case.dz), case.dt, n, case.bc, coriolis_f=1e-4)
        got = run.read(mid)
        for k in FIELDS:
            _same(got[k], want[k], f"{case.shape} {k}")
    run.close()


def test_padded_state_moves_unchanged(ctx):
    """Admission, write, read, image and history of members with padded
    columns: no step in between, so the host's values come back."""
    run = EngineRun(ctx, precision=cuda.PRECISION_REFERENCE)
    states = {}
    for m, shape in enumerate(GRIDS):
        st, base = perturbed_state(_case(shape, OPEN, m), seed=40 + m)
        states[run.admit(_case(shape, OPEN, m), st, base, n_substeps=2)] = st
    for mid, st in states.items():
        got = run.read(mid)
        for k in FIELDS:
            _same(got[k], st[k], f"read {k}")
        st["qr"] = (st["qr"] + np.float32(1e-4)).astype(np.float32)
        run.engine.write(mid, st)
    image = np.empty(run.engine.image_bytes(), np.uint8)
    run.engine.download_image_async(image)
    run.engine.synchronize()
    for mid, views in run.engine.image_views(image).items():
        for k in FIELDS:
            _same(np.ascontiguousarray(views[k]), states[mid][k], f"image {k}")
        frame = np.empty(9 * states[mid]["u"].size, np.float32)
        run.engine.history_async(mid, cuda.HISTORY_CORE, frame)
        run.engine.synchronize()
        frame = frame.reshape(9, *states[mid]["u"].shape)
        _same(np.ascontiguousarray(frame[5]), states[mid]["theta"], "history theta")
        u = states[mid]["u"]
        centre = u.copy()
        centre[1:] = np.float32(0.5) * (u[:-1] + u[1:])
        _same(np.ascontiguousarray(frame[0]), centre, "history u")
    run.close()


@pytest.mark.parametrize("shape", [(68, 72, 64), (66, 70, 64), (70, 67, 65), (37, 29, 45)],
                         ids=["quads", "just-below", "odd", "small"])
def test_fp32_engine_equals_the_per_operation_path(ctx, shape):
    """Both sides of the size from which groups are launched (303,104 cells:
    313,344 and 295,680), and columns the per-operation path cannot group
    (318,920 stored cells in the engine): the same FP32 bits."""
    case = _case(shape, OPEN, 0)
    st, base = cloudy_state(case, seed=3)
    plain = ResidentRun(ctx, case, {k: v.copy() for k, v in st.items()}, base, precision=cuda.PRECISION_FP32,
                        autotune=False)
    run = EngineRun(ctx, precision=cuda.PRECISION_FP32)
    mid = run.admit(case, st, base)
    for _ in range(2):
        plain.step()
    ctx.synchronize()
    run.step(2)
    want, got = plain.download(), run.read(mid)
    for k in FIELDS:
        _same(got[k], want[k], k)
    run.close()


@pytest.mark.parametrize("shape", [(68, 72, 64), (9, 10, 8), (21, 17, 13)], ids=["quads", "small", "odd"])
@pytest.mark.parametrize("bc", [OPEN, CHANNEL, WALLS], ids=["open", "channel", "walls"])
def test_acoustic_loop_and_its_ring(ctx, shape, bc):
    """The per-operation loop with the inner columns closed by the momentum
    pass and the ring around them, the KW78 memory included."""
    import torch

    case = _case(shape, bc, 0)
    st, base = perturbed_state(case, seed=8)
    n, grid = 4, (case.dx, case.dy, case.dz)
    want = {k: v.copy() for k, v in st.items()}
    loop = oracle.Restatement("f32").acoustic_loop(want, base["rho0"], base["p0"], case.dt, n, grid, case.bc)
    ctx.set_precision(cuda.PRECISION_REFERENCE)
    dev = {k: torch.from_numpy(st[k]).cuda() for k in ("u", "v", "w", "rho", "p", "theta")}
    prof = [torch.from_numpy(base[k]).cuda() for k in ("rho0", "p0")]
    mf = [torch.zeros(case.shape, device="cuda") for _ in range(3)]
    wave = torch.zeros(2 * (case.nx + case.ny) * case.nz, device="cuda")
    torch.cuda.synchronize()
    ctx.check(ctx.acoustic_batched(cuda.batched_args(dev, *prof, case.dt / n, n, grid, case.bc, *mf,
                                                     (case.dt / n) / case.dt, None, wave, memory=cuda.MEMORY_DEVICE)))
    ctx.synchronize()
    for k in ("u", "v", "w", "rho", "p"):
        _same(dev[k].cpu().numpy(), want[k], k)
    for a, k in enumerate(("mfx", "mfy", "mfz")):
        _same(mf[a].cpu().numpy(), loop[k], k)
    _same(wave.cpu().numpy(), loop["wave"].astype(np.float32), "wave")


@pytest.mark.parametrize("precision", [cuda.PRECISION_FP32, cuda.PRECISION_REFERENCE], ids=["fp32", "reference"])
def test_members_of_a_crowded_lane_keep_their_bits(ctx, precision):
    """A lane of more than 64 members takes the member-table forms of every
    pass (one cell per thread), a smaller one the constant-bank forms (four
    cells per thread in the FP32 slow pair, and in the acoustic passes of the
    large member's lane): a member's result does not depend on which."""
    shapes = [GRIDS[m % len(GRIDS)] for m in range(65)] + [(70, 67, 65)]
    members = []
    for m, shape in enumerate(shapes):
        case = _case(shape, (OPEN, CHANNEL, WALLS)[m % 3], m)
        members.append((case, *cloudy_state(case, seed=70 + m)))

    def stepped(chosen):
        run = EngineRun(ctx, precision=precision, lanes=1)
        ids = [run.admit(*members[m], coriolis_f=1e-4, n_substeps=3 + m % 3) for m in chosen]
        run.step(2)
        out = {m: run.read(mid) for m, mid in zip(chosen, ids)}
        run.close()
        return out

    together = stepped(range(len(members)))
    apart = {**stepped(range(40)), **stepped(range(40, 65)), **stepped([65])}
    for m, (case, _, _) in enumerate(members):
        for k in FIELDS:
            _same(together[m][k], apart[m][k], f"member {m} {case.shape} {k}")

"""One RK2 step against the oracle at the sizes where the stage kernels change
form: the z-pencil panels (eight FP32 or four FP64 lines; n = 16 has one panel,
48 and 96 no power of two, kxn rarely a multiple of a panel), the y transforms
of one slot (n >= 512) or two, the x chain's tiles of one pair or two and its
batches with a scalar, the overlapped launches (n <= 128 without a scalar), and
a CPU model of the panels' addresses."""
import os
import re
import subprocess

import numpy as np
import pytest


def _eps(prec):
    return 2.0 ** -52 if prec else 2.0 ** -23


def _run(gpu_mod, oracle_mod, n, nc, precs, nu=0.02, rkmethod=2):
    # velmax is about 6 n for this field: a Courant number velmax dt / 2 pi of
    # about 1/4 (step.f refuses numbers above 1)
    dt = 0.25 / n
    o = oracle_mod.Oracle(n, nu, cfl=-1.0, dt=dt, kshift=1, rkmethod=rkmethod)
    if nc:
        o.set_scalar(pr=0.7, grad=(0.3, 0.0, 1.0))
    un = o.field_init(77)
    if nc:
        un[3] = 0.5 * un[0]   # a velocity component is as good a scalar as any
    o.set_state(un)
    assert o.step() == 0
    _, want = o.get_state()
    o.close()
    for prec in precs:
        s = gpu_mod.Solver(n=n, precision=prec, viscos=nu, cfl=-1.0, dt=dt, kshift=1, nc=nc, pr=0.7,
                           grad=(0.3, 0.0, 1.0), rkmethod=rkmethod)
        s.set_state(un)
        assert s.step()["status"] == 0
        got = s.get_state()
        s.close()
        # a transform of n^3 points adds at most about log2(n^3) roundings to a
        # mode, a stage has one there and one back, a step two stages (RK4 four)
        bound = 2 * rkmethod * np.log2(float(n) ** 3) * _eps(prec)
        for v in range(3 + nc):
            err = np.linalg.norm(got[v] - want[v]) / np.linalg.norm(want[v])
            assert err < bound, (n, nc, prec, v, err, bound)


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [0, 1])
@pytest.mark.parametrize("n", [16, 32, 48, 64, 96, 128, 256])
def test_step_against_oracle(gpu_mod, oracle_mod, n, nc):
    _run(gpu_mod, oracle_mod, n, nc, (0, 1))


@pytest.mark.gpu
def test_step_of_512_against_oracle(gpu_mod, oracle_mod):
    _run(gpu_mod, oracle_mod, 512, 0, (0, 1))


@pytest.mark.gpu
def test_step_of_512_with_a_scalar_against_oracle(gpu_mod, oracle_mod):
    """One slot of five fields: 160 threads in FP32, which do not divide a column."""
    _run(gpu_mod, oracle_mod, 512, 1, (0, 1))


@pytest.mark.gpu
def test_rk4_step_of_512_against_oracle(gpu_mod, oracle_mod):
    """advanc_1..4 as epilogues of the one-slot y transforms; four stages."""
    _run(gpu_mod, oracle_mod, 512, 0, (0, 1), rkmethod=4)


@pytest.mark.parametrize("zs,pw", [(2, 8), (1, 4)])
def test_panel_slots_are_a_permutation_without_bank_conflicts(zs, pw):
    """Panel<T, N>: element z of line x at row z / zs, slot x ^ sw(row).  Every
    16-byte slot is used once, and the threads of one phase (16 of 8 bytes, 8 of
    16) reading consecutive z of one line touch every bank once."""
    def sw(rho):
        return rho & 7 if pw == 8 else (rho >> 1) & 3

    def byte(x, z):
        rho = z // zs
        return rho * pw * 16 + ((x ^ sw(rho)) * 16) + (z % zs) * (16 // zs)

    n = 64
    used = sorted(byte(x, z) for x in range(pw) for z in range(n))
    assert used == list(range(0, n // zs * pw * 16, 16 // zs))
    width, phase = 16 // zs, 128 // (16 // zs)
    for x in range(pw):
        for z0 in range(0, n, phase):
            banks = {byte(x, z) % 128 // width for z in range(z0, z0 + phase)}
            assert len(banks) == phase


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
def test_positions_that_are_not_finite_stay_so(gpu_mod, prec):
    """Particles of a run that has blown up: their cells are taken inside the
    grid, their velocities are not finite, and the others are unaffected."""
    n = 32
    pos = 1.0 + n * np.random.default_rng(3).random((64, 3))
    bad = pos.copy()
    bad[::8, 0] = np.nan
    bad[1::8, 2] = np.inf
    out = []
    for p in (pos, bad):
        s = gpu_mod.Solver(n=n, precision=prec, viscos=0.02, cfl=-1.0, dt=0.002)
        s.field_init(5)
        s.particles_set(p)
        for _ in range(2):
            s.particles_advance((0.1, 0.2, 0.3), 0.002)
        out.append(s.particles_get())
        s.close()
    ok = np.isfinite(bad).all(axis=1)
    np.testing.assert_array_equal(out[1][0][ok], out[0][0][ok])
    np.testing.assert_array_equal(out[1][1][ok], out[0][1][ok])
    assert not np.isfinite(out[1][1][~ok]).all(axis=1).any()


def test_layouts_of_the_kernels_header(gpu_mod, tmp_path):
    """tests/stage_layouts.cu, built against the kernels' header: every element of
    a panel has its own place in both orders (z panels and one-slot panels), the
    split addresses of every access of every pass are those places, and the
    shared-memory storage of the tensor-core forms covers their operand tiles."""
    import build as pkg_build
    exe = str(tmp_path / "stage_layouts")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "stage_layouts.cu")
    subprocess.run([pkg_build.NVCC] + pkg_build.FLAGS + ["-O0", "-o", exe, src], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_overlapped_kernels_read_the_steps_data_with_coherent_loads():
    """A kernel launched with launch_dep runs beside the kernel before it, which
    still writes what it reads after dep_wait.  Read-only loads (ld.global.nc:
    __ldg, or a const __restrict__ parameter, for which the compiler may use them)
    are defined only for data that nothing writes during the kernel: tables and
    geometry, not u, un, ub, uz."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = os.path.join(root, "nasa-bluewater-psdns-benchmark-minsky_b200", "csrc", "stage_kernels.cuh")
    with open(path) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    for arg in re.findall(r"__ldg\(\s*([^\s+,)\[]+)", code):
        assert arg.startswith(("g.", "st.")) or arg == "p", arg   # p: ld_step of kernels never overlapped
    assert len(re.findall(r"if constexpr \(!DEP\) return __ldg\(p\);", code)) == len(re.findall(r"__ldg\(p\)", code))
    assert set(re.findall(r"\bld_step<([^;]*?)>\(", code)) == {"dep_launch(N, NC)"}
    kernels = [(name, params) for name, params, body in re.findall(
        r"__global__[^;{]*?\b(k_\w+)\(([^{]*?)\)\s*\{(.*?)\n\}", code, re.S) if re.search(r"dep_wait\(|zfwd_panels<", body)]
    kernels += re.findall(r"\bvoid (zfwd_panels)\(([^{]*?)\)\s*\{", code)
    assert {"k_yinv", "k_zinv", "k_xchain", "k_zfwd", "zfwd_panels", "k_yfwd"} == {name for name, _ in kernels}
    for name, params in kernels:
        for prm in params.split(","):
            if re.search(r"\b(u|un|ub|uz|racc)\b\s*(=|$)", prm.strip()):
                assert not ("const" in prm and "__restrict__" in prm), (name, prm.strip())


@pytest.mark.gpu
@pytest.mark.parametrize("n,nc", [(48, 0), (64, 1), (96, 0), (256, 1), (512, 0)])
@pytest.mark.parametrize("prec,lg", [(0, 46), (1, 470)])
def test_a_step_scales_with_powers_of_two(gpu_mod, n, nc, prec, lg):
    """u -> s u, dt -> dt / s, nu -> s nu (with a scalar and its mean gradient times
    s too) is a symmetry of the step, exact in floating point for a power of two
    while nothing over- or underflows: the squares are below 2^(2 lg + 6), their
    sums over the points of a plane below n^2 of that, and a twiddle pair
    multiplies by at most tan = n / 2 pi on the way: 2^92 2^6 2^18 2^7 < 2^127."""
    sc, out = 2.0 ** lg, []
    for f in (1.0, sc):
        s = gpu_mod.Solver(n=n, precision=prec, viscos=0.02 * f, cfl=-1.0, dt=0.125 / n / f, kshift=1, nc=nc, pr=0.7,
                           grad=(0.3 * f, 0.0, f))
        if not out:
            s.field_init(77)
            un = s.get_state()
            if nc:
                un[3] = 0.5 * un[1]
        s.set_state(f * un)
        assert s.step()["status"] == 0
        out.append(s.get_state() / f)
        s.close()
    np.testing.assert_array_equal(out[0], out[1])

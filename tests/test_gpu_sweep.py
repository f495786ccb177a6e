"""The fast sweep at the edges of its decomposition: tiles of 32 x 8 with two
columns per lane, groups of three planes, chunks of any length.

Fields: rel. L2 to the exact kernel on the same inputs <= 1e-5 (both compute
the same sums in FP32; a few steps apart by some units of 2^-24 each).
Traces: the values the kernel stored, so equal to the fields bit for bit.
"""
import numpy as np
import pytest

from oracle.oracle import rel_l2

pytestmark = pytest.mark.gpu

# (9: one updated point; odd and even ends of a lane's pair; one column or row
# past a full tile; 1, 2 and 0 planes past a full group)
SIZES = [(9, 9, 9), (10, 11, 10), (13, 9, 14), (41, 17, 11), (42, 16, 12), (73, 25, 13),
         (40, 24, 46)]


def inputs(sizes, seed):
    rng = np.random.default_rng(seed)
    shape = sizes[::-1]
    coef = [rng.uniform(-0.5, 0.5, shape).astype(np.float32) for _ in range(6)]
    coef += [rng.uniform(4e6, 9e6, shape).astype(np.float32) for _ in range(4)]
    fields = []
    for _ in range(4):
        f = np.zeros(shape, np.float32)
        f[4:-4, 4:-4, 4:-4] = rng.standard_normal([s - 8 for s in shape])
        fields.append(f)
    return coef, fields


def run(dc, sizes, kernel, medium, coef, fields, src, rec, steps, sponge, d):
    with dc.Simulation(sizes, d, 1e-3, kernel=kernel, medium=medium, device=0) as sim:
        if medium == dc.MEDIUM_PRECOMP:
            sim.set_precomp(coef)
        else:
            sim.set_vpz_vsv(np.sqrt(coef[6]), 0.4 * np.sqrt(coef[7]))
        sim.set_fields(*fields)
        sim.set_source(src, np.linspace(1.0, 2.0, steps + 1))
        if sponge:
            sim.set_sponge(*(np.linspace(0.9, 1.0, n) for n in sizes))
        sim.set_receivers(rec, steps)
        sim.enable_energy(steps)
        sim.run(steps)
        sim.synchronize()
        return sim.get_fields(), sim.traces(steps), sim.energy(steps)


@pytest.mark.parametrize("sponge", [False, True])
@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("sizes", SIZES)
def test_tile_edges(dc, sizes, even, sponge):
    medium = dc.MEDIUM_PRECOMP if even else dc.MEDIUM_VPZ_VSV
    d = (12.5, 12.5, 12.5) if even else (12.5, 10.0, 8.0)
    coef, fields = inputs(sizes, sum(sizes))
    sx, sy, sz = sizes
    # receivers in neighbouring columns, several in one column, both ends of
    # the box, and one at the source
    xs = sorted({4, min(5, sx - 5), sx // 2, sx - 5})
    ys = sorted({4, sy // 2, sy - 5})
    zs = sorted({4, sz // 2, sz - 6, sz - 5} - set(range(4)))
    rec = np.array([x + y * sx + z * sx * sy for z in zs for y in ys for x in xs])
    src = int(rec[len(rec) // 2])
    steps = 3
    got, tr, en = run(dc, sizes, dc.KERNEL_FAST, medium, coef, fields, src, rec, steps, sponge, d)
    want, _, _ = run(dc, sizes, dc.KERNEL_EXACT, medium, coef, fields, src, rec, steps, sponge, d)
    for k in ("pp", "pc", "qp", "qc"):
        assert rel_l2(got[k], want[k]) <= 1e-5, k
    assert np.array_equal(tr[-1], got["pc"].reshape(-1)[rec])
    # the energy of the last step is the sum of squares of the new fields
    total = sum(np.sum(got[k].astype(np.float64) ** 2) for k in ("pc", "qc"))
    assert abs(en[-1] - total) <= 1e-5 * total


@pytest.mark.parametrize("sizes", [(24, 24, 48), (40, 24, 13), (56, 56, 56), (72, 40, 75)])
def test_short_chunks_change_no_bit(dc, monkeypatch, sizes):
    """Small boxes are cut into chunks down to four planes: which CTA computes
    a plane must not show."""
    coef, fields = inputs(sizes, 5)
    sx, sy, sz = sizes
    rec = np.array([sx // 2 + (sy // 2) * sx + z * sx * sy for z in range(4, sz - 4)])
    outs = []
    for chunks in (None, "1", "2"):
        if chunks:
            monkeypatch.setenv("DC_GB300_FAST_ZCHUNKS", chunks)
        with dc.Simulation(sizes, (12.5,) * 3, 1e-3, device=0) as sim:
            sim.set_precomp(coef)
            sim.set_fields(*fields)
            sim.set_source(int(rec[3]), np.linspace(1.0, 2.0, 6))
            sim.set_receivers(rec, 4)
            sim.run(4)
            sim.synchronize()
            outs.append((sim.get_fields(), sim.traces(4)))
    for f, tr in outs[1:]:
        assert all(np.array_equal(f[k], outs[0][0][k]) for k in f)
        assert np.array_equal(tr, outs[0][1])


@pytest.mark.parametrize("medium", ["PRECOMP_F16", "PRECOMP_BF16", "VPZ_VSV"])
@pytest.mark.parametrize("sizes", [(169, 216, 17), (184, 209, 12), (20, 40, 15), (9, 24, 70)])
def test_narrow_last_column(dc, monkeypatch, sizes, medium):
    """Left-over columns in 16 x 16 tiles (1, 16, 12 and 1 of them): the bits of
    the 32 x 16 tiles, which have no such launch; receivers and the source on
    both sides of the cut."""
    form = getattr(dc, "MEDIUM_" + medium)
    coef, fields = inputs(sizes, 6)
    sx, sy, sz = sizes
    cut = 4 + (sx - 8) // 32 * 32
    xs = sorted({max(4, cut - 2), max(4, cut - 1), min(cut, sx - 5), min(cut + 1, sx - 5), sx - 5})
    rec = np.array([x + y * sx + z * sx * sy for z in (4, sz // 2, sz - 5) for y in (4, sy - 5)
                    for x in xs])
    outs = []
    for ty in ("8", "16"):
        monkeypatch.setenv("DC_GB300_FAST_TY", ty)
        with dc.Simulation(sizes, (12.5,) * 3, 1e-3, medium=form, device=0) as sim:
            if medium == "VPZ_VSV":
                sim.set_vpz_vsv(np.sqrt(coef[6]), 0.4 * np.sqrt(coef[7]))
            else:
                sim.set_precomp(coef)
            sim.set_fields(*fields)
            sim.set_source(int(rec[len(xs) + 2]), np.linspace(1.0, 2.0, 6))
            sim.set_sponge(*(np.linspace(0.9, 1.0, n) for n in sizes))
            sim.set_receivers(rec, 5)
            sim.run(3)
            sim.propagate_box((4, 5, 4), (sx - 4, sy - 4, sz - 4))
            sim.run(2)
            sim.synchronize()
            outs.append((sim.get_fields(), sim.traces(5)))
    assert all(np.array_equal(outs[0][0][k], outs[1][0][k]) for k in outs[0][0])
    assert np.array_equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("medium", ["PRECOMP", "PRECOMP_F16", "VPZ_VSV"])
def test_boxes_beside_one_another(dc, medium):
    """Disjoint boxes of a step run beside one another, anything else waits:
    the same calls with a synchronisation after each give the same bits.  The
    overlapping and repeated boxes read what the calls before them wrote."""
    sizes = (88, 72, 64)
    form = getattr(dc, "MEDIUM_" + medium)
    coef, fields = inputs(sizes, 9)
    sx, sy, sz = sizes
    step = [((4, 4, 4), (8, sy - 4, sz - 4)), ((sx - 8, 4, 4), (sx - 4, sy - 4, sz - 4)),
            ((8, 4, 4), (sx - 8, 8, sz - 4)), ((8, sy - 8, 4), (sx - 8, sy - 4, sz - 4)),
            ((8, 8, 4), (sx - 8, sy - 8, 8)), ((8, 8, sz - 8), (sx - 8, sy - 8, sz - 4)),
            ((9, 9, 9), (9, 40, 40)), ((8, 8, 8), (sx - 8, sy - 8, sz - 8))]
    odd = [((7, 9, 10), (40, 41, 30)), ((39, 9, 10), (50, 41, 30)), ((60, 9, 10), (61, 10, 11)),
           ((60, 9, 10), (61, 10, 11)), ((7, 9, 10), (40, 41, 30))]
    outs = []
    for wait in (True, False, False):
        with dc.Simulation(sizes, (12.5,) * 3, 1e-3, medium=form, device=0) as sim:
            if medium == "VPZ_VSV":
                sim.set_vpz_vsv(np.sqrt(coef[6]), 0.4 * np.sqrt(coef[7]))
            else:
                sim.set_precomp(coef)
            sim.set_fields(*fields)
            for _ in range(10):
                for boxes in (step, odd):
                    for b0, b1 in boxes:
                        sim.propagate_box(b0, b1)
                        if wait:
                            sim.synchronize()
                    dc.device_swap_arrays(sim.device_data)
            sim.synchronize()
            outs.append(sim.get_fields())
    for o in outs[1:]:
        assert all(np.array_equal(o[k], outs[0][k]) for k in o)


@pytest.mark.parametrize("medium", [0, 1])
def test_exact_kernel_edges_and_alignment(dc, medium):
    """Two columns per lane give the bits of one column per lane, which takes
    buffers that are not 16-byte aligned: the same boxes through both, over
    ragged sizes."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    for sizes in ((9, 9, 9), (10, 12, 26), (43, 17, 11), (44, 9, 25)):
        sx, sy, sz = sizes
        pitch = (sx + 3) // 4 * 4
        count = pitch * sy * sz
        g = torch.Generator("cuda").manual_seed(sum(sizes))
        per = 10 if medium == 0 else 2
        med = torch.rand(count * per, generator=g, device="cuda") * 0.5
        first = [torch.randn(count * 2 + 2, generator=g, device="cuda") for _ in range(2)]
        outs = []
        for shift in (0, 2):  # floats: 16-byte aligned, and 8 bytes off
            bufs = []
            for f in first:
                b = torch.zeros(count * 2 + 8, device="cuda")
                b[shift:shift + count * 2] = f[:count * 2]
                bufs.append(b)
            cfg = dc.Config(sx, sy, sz, 2.0, 1.5, 1.25, 0.5, dc.KERNEL_EXACT, medium, 0)
            pairs = (C.c_void_p * 2)(*[b.data_ptr() + 4 * shift for b in bufs])
            steps = 3
            energy = np.zeros(steps)
            torch.cuda.synchronize()
            dc.check(dc.lib().dc_gb300_exact_steps_noalloc(
                C.byref(cfg), pairs, med.data_ptr(), steps,
                energy.ctypes.data_as(C.POINTER(C.c_double)), None))
            outs.append([b[shift:shift + count * 2].cpu().numpy() for b in bufs] + [energy])
        a, b = outs
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        assert np.allclose(a[2], b[2], rtol=1e-6, atol=0)


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("sizes", [(40, 24, 46), (73, 41, 29), (104, 56, 75)])
def test_fp32_tile_rows_change_no_bit(dc, monkeypatch, sizes, even):
    """32 x 8 and 32 x 16 tiles of the FP32 form: two CTAs or one per SM, and
    other columns at the edges."""
    d = (12.5, 12.5, 12.5) if even else (12.5, 10.0, 8.0)
    coef, fields = inputs(sizes, 8)
    sx, sy, sz = sizes
    rec = np.array([sx // 2 + y * sx + z * sx * sy for z in (4, sz // 2, sz - 5)
                    for y in (4, sy // 2, sy - 5)])
    outs = []
    for ty in ("8", "16"):
        monkeypatch.setenv("DC_GB300_FAST_TY", ty)
        with dc.Simulation(sizes, d, 1e-3, medium=dc.MEDIUM_PRECOMP, device=0) as sim:
            sim.set_precomp(coef)
            sim.set_fields(*fields)
            sim.set_source(int(rec[4]), np.linspace(1.0, 2.0, 6))
            sim.set_sponge(*(np.linspace(0.9, 1.0, n) for n in sizes))
            sim.set_receivers(rec, 5)
            sim.run(5)
            sim.synchronize()
            outs.append((sim.get_fields(), sim.traces(5)))
    assert all(np.array_equal(outs[0][0][k], outs[1][0][k]) for k in outs[0][0])
    assert np.array_equal(outs[0][1], outs[1][1])
    assert np.abs(outs[0][0]["pc"]).max() > 0


def test_many_boxes_in_a_step(dc):
    """A step in boxes of one point: the bits of one box, and the last calls
    take the host no longer than the first."""
    import time

    sizes = (40, 40, 32)
    sx, sy, sz = sizes
    coef, fields = inputs(sizes, 10)
    out, took = [], []
    for split in (False, True):
        with dc.Simulation(sizes, (12.5,) * 3, 1e-3, device=0) as sim:
            sim.set_precomp(coef)
            sim.set_fields(*fields)
            if not split:
                sim.propagate_box((4, 4, 4), tuple(s - 4 for s in sizes))
            else:
                for z in range(4, sz - 4):
                    for y in range(4, sy - 4):
                        t = time.perf_counter()
                        for x in range(4, sx - 4):
                            sim.propagate_box((x, y, z), (x + 1, y + 1, z + 1))
                        took.append(time.perf_counter() - t)
            sim.synchronize()
            out.append(sim.get_fields())
    assert all(np.array_equal(out[0][k], out[1][k]) for k in out[0])
    # (rows of 32 calls; the first hundred may still fill the launch queue)
    assert np.median(took[-100:]) <= 2.0 * np.median(took[50:150])

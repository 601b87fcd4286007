"""What the decode GEMV's fixed-point activations promise: the range of finite activations they cover, and results that do
not change from one build to the next."""
import zlib

import numpy as np
import pytest

from kraken_b200 import synth

pytestmark = pytest.mark.gpu
SEED = synth.BASE_SEED + 900
FORMATS = [synth.Q8_0, synth.Q4_0, synth.Q4_K, synth.Q6_K, synth.Q5_0, synth.Q5_1, synth.Q5_K, synth.Q2_K, synth.Q3_K, synth.IQ4_NL]
# bytes of a block, offsets of its f16 scales
SCALES = {synth.Q8_0: (34, [0]), synth.Q4_0: (18, [0]), synth.Q5_0: (22, [0]), synth.Q5_1: (24, [0, 2]), synth.IQ4_NL: (18, [0]),
          synth.Q2_K: (84, [80, 82]), synth.Q3_K: (110, [108]), synth.Q4_K: (144, [0, 2]), synth.Q5_K: (176, [0, 2]), synth.Q6_K: (210, [208])}


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("wt", FORMATS)
def test_finite_activations_of_any_size(cuda, oracle, wt):
    """The activation's scale is its largest magnitude over 2^22 - 1, from 1e38 (where a reciprocal of the maximum is a
    subnormal number) down past 1.2e-32 (where 2^22 over the maximum is no f32 any more)."""
    n_out, n_in = 48, 1024
    w = synth.weights(wt, n_out, n_in, SEED, stream=wt)
    size, fields = SCALES[wt]
    blocks = w.reshape(-1, size)
    for at in fields:   # small weights: the sums stay inside the f32 range
        d = (1e-6 * (1.0 + np.arange(len(blocks)) % 7)).astype(np.float16)
        blocks[:, at:at + 2] = d.view(np.uint8).reshape(-1, 2)
    x1 = np.clip(synth.activations(2, n_in, SEED), -3.0, 3.0)
    w64 = oracle.dequant_rows(w, wt, n_out, n_in).astype(np.float64)
    for size in (1e38, 3e37, 1.0, 3e-30, 1e-31, 6e-32, 1e-32, 3e-33):
        x = (x1 * np.float32(size)).astype(np.float32)
        assert np.isfinite(x).all()
        for rows in (1, 2):
            want = x[:rows].astype(np.float64) @ w64.T
            y = cuda.gemv(dev(x[:rows]), dev(w), wt, n_out, n_in).cpu().numpy()
            assert np.abs(want).max() < 1e38
            lim = 2e-6 * np.linalg.norm(w64, axis=1)[None] * np.linalg.norm(x[:rows].astype(np.float64), axis=1)[:, None]
            err = np.abs(y.astype(np.float64) - want)
            assert (err <= lim).all(), (size, rows, float((err / lim).max()))


# crc32 of the f32 results, per format: one row, two rows
RESULTS = {synth.Q8_0: [3056184117, 3582628484], synth.Q4_0: [4275389815, 4277281545], synth.Q4_K: [3915479935, 2426236879],
           synth.Q6_K: [607611225, 2896286947], synth.Q5_0: [4107378900, 2160153247], synth.Q5_1: [2911803218, 1148909278],
           synth.Q5_K: [765817051, 716160757], synth.Q2_K: [2228023986, 3771803034], synth.Q3_K: [3856678096, 3514639972],
           synth.IQ4_NL: [2476352332, 1264748544]}


def results(cuda, wt):
    n_out, n_in = 96, 4096
    w = dev(synth.weights(wt, n_out, n_in, SEED + 1, stream=wt))
    i = np.arange(2 * n_in, dtype=np.uint64)
    x = dev(((i * 2654435761 % (1 << 32)).astype(np.float64) / (1 << 31) - 1.0).astype(np.float32).reshape(2, n_in))
    return [zlib.crc32(cuda.gemv(x[:rows], w, wt, n_out, n_in).cpu().numpy().tobytes()) for rows in (1, 2)]


@pytest.mark.parametrize("wt", FORMATS)
def test_one_and_two_row_results_keep_their_bits(cuda, wt):
    """A logit of 250 has steps of 1.5e-5, and the mass over a vocabulary takes exp() of such numbers: a different order of
    the final f32 sums, each as good as the other, shows there as 2e-5. So the order stays."""
    assert results(cuda, wt) == RESULTS[wt]


# (K = 11008 leaves a ring of few stages beside eight prepared rows; K = 2080 and 5120 are rows that start at any even address)
@pytest.mark.parametrize("wt, n_out, n_in", [(synth.Q6_K, 3000, 11008), (synth.Q3_K, 3000, 5120), (synth.Q8_0, 3000, 2080), (synth.Q8_0, 5000, 4096),
                                             (synth.Q4_K, 5000, 11008), (synth.Q4_0, 5000, 4096)])
def test_stages_are_refilled_only_once_read(cuda, wt, n_out, n_in):
    """The same call over and over, between calls that fill the ring with other bytes: same bits, and the right sums."""
    import torch
    w, other = (dev(synth.weights(wt, n_out, n_in, SEED + 2 + i, stream=wt)) for i in range(2))
    w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
    for rows in (1, 2, 3, 5, 8):
        x = dev(synth.activations(rows, n_in, SEED + rows))
        first = cuda.gemv(x, w, wt, n_out, n_in)
        lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None]
        assert ((first.double() - x.double() @ w64.T).abs() <= lim).all()
        for _ in range(40):
            cuda.gemv(x, other, wt, n_out, n_in)
            assert torch.equal(cuda.gemv(x, w, wt, n_out, n_in), first)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("wt", [synth.Q8_0, synth.Q4_0, synth.Q5_0, synth.Q5_1, synth.IQ4_NL])
def test_rows_of_odd_block_counts_are_as_exact_as_f32(cuda, wt, outliers):
    """K not a multiple of 256. The warp-per-row kernel, which such shapes took before, multiplies in f32: over these
    very inputs its worst distance from the f64 sums (2-norm) is 1.7e-7 for Q5_1 and 1.4e-7 for the others, with activations
    three hundred times as large in every 97th place as without."""
    worst = 0.0
    for n_out, n_in in ((256, 288), (512, 2080), (416, 2912), (300, 5600), (300, 9248)):
        w = dev(synth.weights(wt, n_out, n_in, SEED + 4, stream=wt))
        w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
        for rows in (1, 2, 3, 5, 7, 8, 37):
            x = synth.activations(rows, n_in, SEED + rows)
            if outliers:
                x[:, 5::97] *= 300.0
            x = dev(x)
            y = cuda.gemv(x, w, wt, n_out, n_in) if rows <= 8 else cuda.gemm(x, w, wt, n_out, n_in)
            want = x.double() @ w64.T
            worst = max(worst, ((y.double() - want).norm() / want.norm()).item())
    assert worst <= (1.7e-7 if wt == synth.Q5_1 else 1.4e-7)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", [synth.Q8_0, synth.Q4_0, synth.Q5_0, synth.Q5_1, synth.IQ4_NL])
def test_rows_of_odd_block_counts_keep_infinities(cuda, wt):
    """K not a multiple of 256: an infinite activation gives what f32 arithmetic gives, and only in its own row."""
    import torch
    n_out, n_in = 100, 2080
    w = dev(synth.weights(wt, n_out, n_in, SEED + 5, stream=wt))
    w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
    for rows in (1, 2, 4, 8, 11):
        x = dev(synth.activations(rows, n_in, SEED + rows))
        x[rows // 2, 777] = float("-inf")
        if rows > 2:
            x[0, 2079] = float("nan")
        want = x.double() @ w64.T
        got = cuda.gemv(x, w, wt, n_out, n_in) if rows <= 8 else cuda.gemm(x, w, wt, n_out, n_in)
        assert torch.isinf(want[rows // 2]).any()
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        assert torch.equal(torch.sign(got[torch.isinf(got)]).double(), torch.sign(want[torch.isinf(want)]))
        fine = torch.isfinite(want)
        assert (got[fine].double() - want[fine]).norm() <= 2e-7 * want[fine].norm()
    # the gate/up fold: silu(gate) of an infinite gate
    x = dev(synth.activations(1, n_in, SEED))[0]
    x[777] = float("inf")
    got = cuda.gemv_group([x, x], [w, w], [wt, wt], [n_out, n_out], n_in, fuse_silu_pair=True)[0]
    gate = x.double() @ w64.T
    want = gate / (1.0 + torch.exp(-gate)) * gate
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))


# (a box holds a stage's part of 16 rows and up to 16 bytes more of each: one stage and several, whole and clipped by the row's end,
# stacked tiles; rows clipped by the matrix's end; launches on either side of the rules by tiles, of 74, 148, 222 and 296)
@pytest.mark.parametrize("wt, widths", [(synth.Q8_0, (256, 512, 1024, 2304, 4096, 11008)), (synth.Q2_K, (1024, 3072, 8192)),
                                        (synth.Q3_K, (2048, 6144)), (synth.Q5_1, (256, 768, 2304, 4096))])
def test_stages_in_one_box_of_padded_rows(cuda, wt, widths):
    import torch
    for n_in in widths:
        for n_out in (1, 15, 33, 1185, 2367, 2369, 3553, 4737):
            w = dev(synth.weights(wt, n_out, n_in, SEED + 7, stream=wt))
            w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
            for rows in (1, 2, 4, 7):
                x = dev(synth.activations(rows, n_in, SEED + rows))
                y = cuda.gemv(x, w, wt, n_out, n_in)
                # the bound of test_finite_activations_of_any_size: 22 bits of x against its largest value, twice over
                lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None]
                assert ((y.double() - x.double() @ w64.T).abs() <= lim).all(), (n_in, n_out, rows)
    assert cuda.device_status() == 0


# Row copies again where CTAs have as many tiles (74 SMs' and 148's worth of 16 rows, twice and thrice that and more), on either side
@pytest.mark.parametrize("wt, n_in, n_outs, row_counts", [
    (synth.Q5_1, 1280, (8500, 9216), (1, 2)), (synth.Q5_1, 4096, (4600, 4736, 9216, 14208), (1, 2, 3, 5, 6)), (synth.Q5_1, 5632, (4736, 18432), (2, 4)),
    (synth.Q8_0, 1024, (4800, 8192, 9472, 14224), (2,)), (synth.Q8_0, 2048, (5632, 8192, 14000, 14224), (2,)), (synth.Q8_0, 4096, (4144, 4145, 4700), (1,)),
    (synth.Q2_K, 2048, (1200, 2368, 2369), (1, 2)), (synth.Q3_K, 2048, (1200, 2368, 2369), (1, 2))])
def test_row_copies_where_tiles_come_out_even(cuda, wt, n_in, n_outs, row_counts):
    import torch
    for n_out in n_outs:
        w = dev(synth.weights(wt, n_out, n_in, SEED + 19, stream=wt))
        w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
        for rows in row_counts:
            x = dev(synth.activations(rows, n_in, SEED + rows))
            y = cuda.gemv(x, w, wt, n_out, n_in)
            # as in test_stages_in_one_box_of_padded_rows
            lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None]
            assert ((y.double() - x.double() @ w64.T).abs() <= lim).all(), (n_out, rows)
    assert cuda.device_status() == 0


# Rows that are not 16-byte multiples go in tiles of rows 2, 4 or 8 apart: K = 32, 64 and 128 times odd numbers (Q8_0, Q4_0, IQ4_NL, Q5_0),
# any K off a multiple of 2048 (Q6_K that long or that odd, Q3_K) or 1024 (Q2_K); matrices of fewer rows than that, of parts of
# tiles, and on either side of a tile for every SM
@pytest.mark.parametrize("wt, widths", [(synth.Q8_0, (288, 544, 1056, 2112, 2176)), (synth.Q4_0, (2080, 2112, 2176)), (synth.Q5_0, (2080, 2176)),
                                        (synth.Q5_1, (2080, 2112)), (synth.IQ4_NL, (2080,)), (synth.Q6_K, (4352, 4864, 5120, 11008)), (synth.Q3_K, (256, 512, 1024, 2304)),
                                        (synth.Q2_K, (256, 512, 2304))])
def test_ragged_rows_in_tiles_of_a_phase(cuda, wt, widths):
    import torch
    for n_in in widths:
        for n_out in (1, 7, 9, 129, 600, 2367, 2500, 4739):
            w = dev(synth.weights(wt, n_out, n_in, SEED + 8, stream=wt))
            w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
            for rows in (1, 2, 3, 8):
                x = dev(synth.activations(rows, n_in, SEED + rows))
                base = torch.randn((rows, n_out), device="cuda")
                y = cuda.gemv(x, w, wt, n_out, n_in, out=base.clone(), accumulate=True)
                # as in test_stages_in_one_box_of_padded_rows, and the rounding of the sum with the old value
                lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None] + 1e-6 * base.abs()
                assert ((y.double() - base - x.double() @ w64.T).abs() <= lim).all(), (n_in, n_out, rows)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt, n_in", [(synth.Q8_0, 2080), (synth.Q5_1, 2080), (synth.Q6_K, 2304), (synth.Q3_K, 5120), (synth.Q2_K, 2304)])
def test_few_ragged_rows_on_either_side_of_the_dealing(cuda, wt, n_in):
    """Whole tiles (of 8, 4 or 2 phases) up to nine twentieths of 148 SMs, ten to fourteen rows on every SM beyond."""
    import torch
    for n_out in (232, 263, 416, 591, 1024, 1025, 1056, 1057, 1153):
        w = dev(synth.weights(wt, n_out, n_in, SEED + 17, stream=wt))
        w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
        for rows in (1, 2):
            x = dev(synth.activations(rows, n_in, SEED + rows))
            base = torch.randn((rows, n_out), device="cuda")
            y = cuda.gemv(x, w, wt, n_out, n_in, out=base.clone(), accumulate=True)
            # as in test_ragged_rows_in_tiles_of_a_phase
            lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None] + 1e-6 * base.abs()
            assert ((y.double() - base - x.double() @ w64.T).abs() <= lim).all(), (n_out, rows)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt, n_in", [(synth.Q8_0, 2080), (synth.Q6_K, 5120), (synth.Q3_K, 2304)])
def test_ragged_rows_of_groups(cuda, wt, n_in):
    """Three matrices of eight phases still have a tensor map each, four are copied row by row; pairs; a group as Backend sends it."""
    import torch
    x = dev(synth.activations(1, n_in, SEED))[0]
    for sizes in ((2080, 416, 417), (300, 5, 33, 1000), (9,)):
        ws = [dev(synth.weights(wt, n, n_in, SEED + 9 + i, stream=wt)) for i, n in enumerate(sizes)]
        got = cuda.gemv_group([x] * len(sizes), ws, [wt] * len(sizes), list(sizes), n_in)
        for n, w, y in zip(sizes, ws, got):
            w64 = cuda.dequant_rows(w, wt, n, n_in).double()
            assert ((y.double() - w64 @ x.double()).abs() <= 2e-6 * w64.norm(dim=1) * x.double().norm()).all()
    for n in (33, 3000):
        w, v = (dev(synth.weights(wt, n, n_in, SEED + 20 + i, stream=wt)) for i in range(2))
        got = cuda.gemv_group([x, x], [w, v], [wt, wt], [n, n], n_in, fuse_silu_pair=True)[0].double()
        g, u = (cuda.dequant_rows(m, wt, n, n_in).double() @ x.double() for m in (w, v))
        want = g / (1.0 + torch.exp(-g)) * u
        assert (got - want).norm() <= 2e-6 * want.norm()
    assert cuda.device_status() == 0


# One and two rows of many stages go to two groups of warps that take a tile's stages in turn: a tile for an SM at most beyond 5120
# values (129 tiles up to 8192), and any number where half an SM has no room for the ring
@pytest.mark.parametrize("wt", FORMATS)
def test_one_and_two_rows_with_stages_in_turn(cuda, wt):
    import torch
    widths = (5152, 5376, 8192, 11008, 14336) if SCALES[wt][0] < 84 else (5376, 8192, 11008, 14336)
    for n_in in widths:
        for n_out in (5, 600, 2064, 2065, 2368, 2369, 4739):
            w = dev(synth.weights(wt, n_out, n_in, SEED + 10, stream=wt))
            w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
            for rows in (1, 2):
                x = dev(synth.activations(rows, n_in, SEED + rows))
                base = torch.randn((rows, n_out), device="cuda")
                y = cuda.gemv(x, w, wt, n_out, n_in, out=base.clone(), accumulate=True)
                lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None] + 1e-6 * base.abs()
                assert ((y.double() - base - x.double() @ w64.T).abs() <= lim).all(), (n_in, n_out, rows)
    # groups of two activations, and gate/up pairs
    n_in, sizes = 11008, (700, 33)
    x, z = dev(synth.activations(2, n_in, SEED))
    ws = [dev(synth.weights(wt, n, n_in, SEED + 11 + i, stream=wt)) for i, n in enumerate(sizes)]
    for v, n, w, y in zip((x, z), sizes, ws, cuda.gemv_group([x, z], ws, [wt] * 2, list(sizes), n_in)):
        w64 = cuda.dequant_rows(w, wt, n, n_in).double()
        assert ((y.double() - w64 @ v.double()).abs() <= 2e-6 * w64.norm(dim=1) * v.double().norm()).all()
    pair = [dev(synth.weights(wt, 900, n_in, SEED + 13 + i, stream=wt)) for i in range(2)]
    got = cuda.gemv_group([x, x], pair, [wt, wt], [900, 900], n_in, fuse_silu_pair=True)[0].double()
    g, u = (cuda.dequant_rows(m, wt, 900, n_in).double() @ x.double() for m in pair)
    want = g / (1.0 + torch.exp(-g)) * u
    assert (got - want).norm() <= 2e-6 * want.norm()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", FORMATS)
def test_slices_of_a_sharded_head_keep_the_bits_of_the_whole(cuda, wt):
    """krk_cuda_gemv_allgather, a slice at a time into one row: the form, and with it the order of sums, goes by the rows of the whole head
    (of 296 tiles, where a slice has 148 or fewer, and of one tile for an SM)."""
    import torch
    for n_in in (5376, 8192, 8960):
        for n_out, cuts in ((4736, (0, 2368, 3000, 4736)), (2000, (0, 1000, 2000))):
            w = dev(synth.weights(wt, n_out, n_in, SEED + 16, stream=wt))
            per_row = w.numel() // n_out
            for rows in (1, 2, 3):
                x = dev(synth.activations(rows, n_in, SEED + rows))
                full, flags = torch.zeros((rows, n_out), device="cuda"), torch.zeros(3, dtype=torch.int32, device="cuda")
                for step, (lo, hi) in enumerate(zip(cuts, cuts[1:])):
                    cuda.gemv_allgather([full.data_ptr()], [flags.data_ptr()], 0, step + 1, lo, n_out, x, w.view(-1)[lo * per_row:hi * per_row], wt, hi - lo, n_in)
                assert torch.equal(full, cuda.gemv(x, w, wt, n_out, n_in)), (n_in, n_out, rows)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", [synth.Q4_K, synth.Q6_K, synth.Q8_0])
def test_routed_experts_of_wide_activations(cuda, wt):
    """The same two groups behind a device-side table of matrices."""
    import torch
    n_embd, n_ff, n_exp = 14336, 256, 4
    gate, up = (dev(synth.weights(wt, n_exp * n_ff, n_embd, SEED + 30 + i, stream=wt)) for i in range(2))
    down = dev(synth.weights(wt, n_exp * n_embd, n_ff, SEED + 32, stream=wt))
    bank = cuda.make_bank(gate, up, down, wt, wt, n_exp, 0, n_embd, n_ff)
    G, U = (cuda.dequant_rows(m, wt, n_exp * n_ff, n_embd).double().view(n_exp, n_ff, n_embd) for m in (gate, up))
    D = cuda.dequant_rows(down, wt, n_exp * n_embd, n_ff).double().view(n_exp, n_embd, n_ff)
    for rows in (1, 2, 5):
        x = dev(synth.activations(rows, n_embd, SEED + rows))
        ids, wts = cuda.route(dev(synth.activations(rows, n_exp, SEED, stream=7)), 2)
        y = cuda.moe_ffn(x, ids, wts, bank).double()
        want = torch.zeros_like(y)
        for r in range(rows):
            for e, c in zip(ids[r].tolist(), wts[r].double()):
                g, u = G[e] @ x[r].double(), U[e] @ x[r].double()
                want[r] += c * (D[e] @ (g / (1.0 + torch.exp(-g)) * u))
        assert (y - want).norm() <= 4e-6 * want.norm(), rows
    assert cuda.device_status() == 0


@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("wt", FORMATS)
def test_rows_without_room_are_as_exact_as_f32(cuda, wt, outliers):
    """K a multiple of 256 and so many activation rows that their limbs leave no room for a ring: parts of them, with four limbs. The
    warp-per-row kernel, which such shapes took before, is 1.4e-7 to 1.64e-7 from the f64 sums over such inputs."""
    import torch
    for n_out, n_in in ((700, 14592), (33, 14336), (513, 16640), (530, 20480)):   # (no format has room for five rows)
        w = dev(synth.weights(wt, n_out, n_in, SEED + 14, stream=wt))
        w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
        for rows in (5, 6, 7, 8):
            x = synth.activations(rows, n_in, SEED + rows)
            if outliers:
                x[:, 5::97] *= 300.0
            x = dev(x)
            base = torch.zeros((rows, n_out), device="cuda")
            y = cuda.gemv(x, w, wt, n_out, n_in, out=base, accumulate=True)
            want = x.double() @ w64.T
            err = ((y.double() - want).norm() / want.norm()).item()
            assert err <= 1.64e-7, (n_in, rows, err)
    # an infinite activation gives what f32 arithmetic gives, and only in its own row
    n_out, n_in, rows = 40, 14336, 7
    w = dev(synth.weights(wt, n_out, n_in, SEED + 15, stream=wt))
    w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
    x = dev(synth.activations(rows, n_in, SEED))
    x[3, 777], x[0, 5] = float("-inf"), float("nan")
    want, got = x.double() @ w64.T, cuda.gemv(x, w, wt, n_out, n_in)
    assert torch.isinf(want[3]).any()
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine = torch.isfinite(want)
    assert (got[fine].double() - want[fine]).norm() <= 2e-7 * want[fine].norm()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("wt", FORMATS)
def test_two_to_four_rows_without_room(cuda, wt, outliers):
    """The widest rows: two, three and four of them in parts of two and one, added onto what is there. The warp-per-row kernel, which
    such shapes took before, is at worst this far from the f64 sums over such inputs (16128, 21504 and 32512 values; the fewest weight
    rows leave the most to chance); and the rounding of the last sum."""
    import torch
    for n_in, rows, bound in ((16128, 4, 1.71e-7), (21504, 3, 1.88e-7), (32512, 2, 2.11e-7)):   # (beyond what any format has room for)
        for n_out, worst in ((33, 2.46e-7), (530, bound)):
            w = dev(synth.weights(wt, n_out, n_in, SEED + 21, stream=wt))
            x = synth.activations(rows, n_in, SEED + rows)
            if outliers:
                x[:, 5::97] *= 300.0
            x = dev(x)
            base = torch.randn((rows, n_out), device="cuda")
            got = cuda.gemv(x, w, wt, n_out, n_in, out=base.clone(), accumulate=True).double()
            want = x.double() @ cuda.dequant_rows(w, wt, n_out, n_in).double().T
            assert (got - base - want).norm() <= worst * want.norm() + 2.0 ** -24 * got.norm(), (n_in, rows, n_out)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", [synth.Q8_0, synth.IQ4_NL, synth.Q5_1])
def test_rows_without_room_add_no_error_block_by_block(cuda, wt):
    """The 32-value formats at the widths where a warp adds the most blocks: the mean of eight errors is that of sums by unit (1.0e-7 to
    1.1e-7 here), below what adding block by block gives (1.38e-7 to 1.45e-7; the warp-per-row kernel 1.33e-7 to 1.42e-7)."""
    errs = []
    for i in range(8):
        n_out, n_in, rows = 530, 12544, 6
        w = dev(synth.weights(wt, n_out, n_in, 900 + i, stream=wt))
        x = dev(synth.activations(rows, n_in, 77 + i))
        want = x.double() @ cuda.dequant_rows(w, wt, n_out, n_in).double().T
        errs.append(((cuda.gemv(x, w, wt, n_out, n_in).double() - want).norm() / want.norm()).item())
    assert np.mean(errs) <= 1.25e-7, errs


@pytest.mark.parametrize("wt", [synth.Q4_K, synth.Q2_K, synth.Q6_K, synth.Q8_0, synth.Q5_1])
def test_rows_without_room_in_groups_pairs_and_residuals(cuda, wt):
    """As a model's layer sends them: two matrices of one activation, a gate/up pair (silu has a slope of 1.1 at most), a projection
    onto the residual."""
    import torch
    be = cuda.Backend(0)
    for n_in in (12544, 14336):   # (no format has room for five rows)
        ws = [dev(synth.weights(wt, n, n_in, SEED + 22 + i, stream=wt)) for i, n in enumerate((700, 1033, 1033))]
        w64 = [cuda.dequant_rows(w, wt, n, n_in).double() for w, n in zip(ws, (700, 1033, 1033))]
        for rows in (5, 6, 8):
            x = dev(synth.activations(rows, n_in, SEED + rows))
            want = [x.double() @ m.T for m in w64]
            ys = [torch.full((rows, n), 7.0, device="cuda") for n in (700, 1033)]
            torch.cuda.synchronize()
            ran, _ = be.gemm_group([y.data_ptr() for y in ys], x.data_ptr(), [w.data_ptr() for w in ws[:2]], wt, [700, 1033], n_in, rows=rows)
            be.sync()
            assert ran
            for y, v in zip(ys, want):
                assert (y.double() - v).norm() <= 1.64e-7 * v.norm(), (n_in, rows)
            ys = [torch.full((rows, 1033), 7.0, device="cuda") for _ in range(2)]
            torch.cuda.synchronize()
            ran, fused = be.gemm_group([y.data_ptr() for y in ys], x.data_ptr(), [w.data_ptr() for w in ws[1:]], wt, [1033] * 2, n_in, rows=rows, silu=True)
            be.sync()
            assert ran
            if fused:
                v = want[1] / (1.0 + torch.exp(-want[1])) * want[2]
                lim = 2e-6 * x.double().norm(dim=1)[:, None] * (1.1 * w64[1].norm(dim=1)[None] * want[2].abs() + w64[2].norm(dim=1)[None] * want[1].abs()) + 1e-6 * v.abs()
                assert ((ys[0].double() - v).abs() <= lim).all(), (n_in, rows)
            base = torch.randn((rows, 700), device="cuda")
            y = base.clone()
            torch.cuda.synchronize()
            assert be.gemm_accumulate(y.data_ptr(), x.data_ptr(), ws[0].data_ptr(), wt, 700, n_in, rows)
            be.sync()
            assert (y.double() - base - want[0]).norm() <= 1.64e-7 * want[0].norm() + 2.0 ** -24 * y.double().norm(), (n_in, rows)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("n_out", [4736, 4737, 5003])
def test_q8_0_three_and_four_rows_across_the_change_of_form(cuda, n_out):
    """Up to two tiles of 16 weight rows per SM (148: 4736 rows) two consumer groups share a CTA, beyond that every CTA has one."""
    import torch
    for n_in in (1024, 4096):
        w = dev(synth.weights(synth.Q8_0, n_out, n_in, SEED + 6, stream=1))
        w64 = cuda.dequant_rows(w, synth.Q8_0, n_out, n_in).double()
        for rows in (2, 3, 4, 5):
            x = dev(synth.activations(rows, n_in, SEED + rows))
            base = torch.randn((rows, n_out), device="cuda")
            y = cuda.gemv(x, w, synth.Q8_0, n_out, n_in, out=base.clone(), accumulate=True)
            lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None] + 1e-6 * base.abs()
            assert ((y.double() - base.double() - x.double() @ w64.T).abs() <= lim).all()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("n_in, tiles", [(768, (3, 5, 14)), (1024, (2, 3, 5, 14)), (4096, (2, 6))])
def test_q8_0_three_and_four_rows_of_one_group(cuda, n_in, tiles):
    """Two consumer groups share a CTA up to six tiles of 16 weight rows per SM at three rows and everywhere at four; up to 1024 values
    up to three at three rows, five at four (three below 1024). Beyond, every CTA has one group, and two share an SM; up to 1024 values
    stages come as row copies from five to fourteen tiles per SM."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n_out in sorted({16 * sms * t + more for t in tiles for more in (0, 1, 267)}):
        w = dev(synth.weights(synth.Q8_0, n_out, n_in, SEED + 6, stream=1))
        w64 = cuda.dequant_rows(w, synth.Q8_0, n_out, n_in).double()
        for rows in (2, 3, 4, 5):
            x = dev(synth.activations(rows, n_in, SEED + rows))
            base = torch.randn((rows, n_out), device="cuda")
            y = cuda.gemv(x, w, synth.Q8_0, n_out, n_in, out=base.clone(), accumulate=True)
            lim = 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None] + 1e-6 * base.abs()
            assert ((y.double() - base.double() - x.double() @ w64.T).abs() <= lim).all(), (n_out, rows)
    assert cuda.device_status() == 0


def test_q8_0_three_rows_of_one_group_in_a_launch_of_two_matrices(cuda):
    import torch
    n_in, rows, sizes = 4096, 3, (9000, 6001)   # 938 tiles: beyond six per SM together
    x = dev(synth.activations(rows, n_in, SEED))
    ws = [dev(synth.weights(synth.Q8_0, n, n_in, SEED + 18 + i, stream=i)) for i, n in enumerate(sizes)]
    ys = [torch.zeros((rows, n), device="cuda") for n in sizes]
    be = cuda.Backend(0)
    torch.cuda.synchronize()
    ran, _ = be.gemm_group([y.data_ptr() for y in ys], x.data_ptr(), [w.data_ptr() for w in ws], synth.Q8_0, list(sizes), n_in, rows=rows)
    be.sync()
    assert ran
    for n, w, y in zip(sizes, ws, ys):
        w64 = cuda.dequant_rows(w, synth.Q8_0, n, n_in).double()
        assert ((y.double() - x.double() @ w64.T).abs() <= 2e-6 * w64.norm(dim=1)[None] * x.double().norm(dim=1)[:, None]).all()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", [synth.Q8_0, synth.Q4_0, synth.Q5_1])
def test_rows_of_odd_block_counts_on_either_kernel(cuda, wt):
    """The lines between the streaming and the warp-per-row kernel, K not a multiple of 256: K = 1024 from 512 weight rows on
    (Q5_1: 2048 below eight rows per SM), and wide activations of many rows, in two launches or not."""
    for n_out, n_in, row_counts in ((511, 992, (1, 3, 8)), (512, 992, (1, 3, 8)), (512, 1056, (1, 8)), (1183, 2016, (2, 5)), (1184, 2016, (2, 5)),
                                    (100, 11232, (5, 6, 7, 8)), (1200, 11232, (5, 8))):
        w = dev(synth.weights(wt, n_out, n_in, SEED + 7, stream=wt))
        w64 = cuda.dequant_rows(w, wt, n_out, n_in).double()
        for rows in row_counts:
            x = dev(synth.activations(rows, n_in, SEED + rows))
            want = x.double() @ w64.T
            for _ in range(2):
                y = cuda.gemv(x, w, wt, n_out, n_in)
                # (the bound of the f32 kernel's distance above, for its longer rows too)
                assert ((y.double() - want).norm() / want.norm()).item() <= 3e-7, (n_out, n_in, rows)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("wt", FORMATS)
@pytest.mark.parametrize("n_in", [2304, 4352, 6656, 11008, 12544])
def test_rows_of_many_slices(cuda, oracle, wt, n_in):
    """A warp prepares one to seven slices of every activation row (held, in one batch of loads, in a second; six of the widest rows go
    to the warp-per-row kernel in most formats). 22 bits of the largest activation of a warp's slices
    (about four sigma here) leave 4 * 2^-22 / sqrt(12) a value, 2.8e-7 of the norms' product for a result; seven times that."""
    n_out = 80
    w = synth.weights(wt, n_out, n_in, SEED + 2, stream=wt)
    w64 = oracle.dequant_rows(w, wt, n_out, n_in).astype(np.float64)
    x = synth.activations(6, n_in, SEED + 3)
    x[1] *= 1e-3
    for rows in (1, 2, 3, 4, 6):
        y = cuda.gemv(dev(x[:rows]), dev(w), wt, n_out, n_in).cpu().numpy()
        x64 = x[:rows].astype(np.float64)
        lim = 2e-6 * np.linalg.norm(w64, axis=1)[None] * np.linalg.norm(x64, axis=1)[:, None]
        assert (np.abs(y.reshape(rows, n_out) - x64 @ w64.T) <= lim).all(), rows


@pytest.mark.parametrize("n_in, n_out, row_counts", [(11008, 7201, (3, 4)), (6656, 7201, (4, 5, 6)), (8960, 4801, (3, 5)), (12544, 100, (4,)), (10496, 1000, (5,))])
def test_stages_of_a_tile_in_turn(cuda, n_in, n_out, row_counts):
    """Ragged Q6_K rows whose ring does not hold two tiles: both consumer groups multiply every tile, each through slots of its own
    (two at three and four rows, one beyond), which a CTA's third and fourth tile meet again, an odd number of stages later too;
    the last two shapes are one tile a CTA in a ring of two stages. The bound is that of test_rows_of_many_slices; silu has a slope
    of 1.1 at most."""
    import torch
    wt = synth.Q6_K
    w, other = (dev(synth.weights(wt, n_out, n_in, SEED + 8, stream=20 + i)) for i in range(2))
    w64, other64 = (cuda.dequant_rows(m, wt, n_out, n_in).double() for m in (w, other))
    be = cuda.Backend(0)
    for rows in row_counts:
        x = dev(synth.activations(rows, n_in, SEED + rows))
        norms = x.double().norm(dim=1)[:, None]
        want, lim = x.double() @ w64.T, 2e-6 * w64.norm(dim=1)[None] * norms
        before = cuda.family_count(cuda.FAMILY_GEMV_STREAM)
        first = cuda.gemv(x, w, wt, n_out, n_in)
        assert cuda.family_count(cuda.FAMILY_GEMV_STREAM) == before + 1
        assert ((first.double() - want).abs() <= lim).all(), rows
        for _ in range(10):
            cuda.gemv(x, other, wt, n_out, n_in)
            assert torch.equal(cuda.gemv(x, w, wt, n_out, n_in), first)
        base = torch.randn((rows, n_out), device="cuda")
        got = cuda.gemv(x, w, wt, n_out, n_in, out=base.clone(), accumulate=True)
        assert torch.equal(got, base + first)
        # several matrices in one launch, and the gate/up fold
        outs = [torch.empty((rows, n_out), device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        before = cuda.family_count(cuda.FAMILY_GEMV_STREAM)
        ran, _ = be.gemm_group([o.data_ptr() for o in outs], x.data_ptr(), [m.data_ptr() for m in (w, other, w)], wt, [n_out] * 3, n_in, rows=rows)
        torch.cuda.synchronize()
        assert ran and cuda.family_count(cuda.FAMILY_GEMV_STREAM) == before + 1
        up, up_lim = x.double() @ other64.T, 2e-6 * other64.norm(dim=1)[None] * norms
        assert ((outs[0].double() - want).abs() <= lim).all() and torch.equal(outs[2], outs[0])
        assert ((outs[1].double() - up).abs() <= up_lim).all()
        ran, fused = be.gemm_group([o.data_ptr() for o in outs[:2]], x.data_ptr(), [m.data_ptr() for m in (w, other)], wt, [n_out] * 2, n_in, rows=rows,
                                   silu=True)
        torch.cuda.synchronize()
        assert ran and fused
        silu = want / (1.0 + torch.exp(-want))
        assert ((outs[0].double() - silu * up).abs() <= 1.1 * lim * (up.abs() + up_lim) + silu.abs() * up_lim + 1e-6 * (silu * up).abs()).all()
    be.close()
    assert cuda.device_status() == 0

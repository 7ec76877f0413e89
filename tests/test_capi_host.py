"""Host-side checks that need no GPU: the C ABI library loads and exports every
symbol the header declares, and its host logic (ConvParams algebra, planner,
error reporting) agrees with the oracle and with the reference's messages."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import oracle
from oracle import ConvSpec
from poplibs_b200 import capi
from test_oracle import OUTPUT_DIM_TABLE, RANGE_TABLE, random_spec

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "poplibs_b200.h")).read()
    return sorted(set(re.findall(r"PLB_API[^;(]*?\b(plb_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    lib = capi.lib()
    names = declared_symbols()
    assert len(names) >= 30
    for name in names:
        assert hasattr(lib, name), f"{name} declared in include/poplibs_b200.h but not exported"
    assert sorted(capi.SYMBOLS) == names
    assert b"sm_100a" in lib.plb_version()


def params_from_spec(spec: ConvSpec) -> capi.ConvParams:
    return capi.ConvParams.make(spec.batch, spec.field, spec.kernel, spec.in_chans, spec.out_chans,
                                spec.groups, **spec.normalised_transforms()) \
        if hasattr(spec, "normalised_transforms") else _params_from_spec(spec)


def _params_from_spec(spec):
    n = spec.normalised()
    n.pop("field"), n.pop("kernel")
    return capi.ConvParams.make(spec.batch, spec.field, spec.kernel, spec.in_chans, spec.out_chans,
                                spec.groups, **n)


def test_input_index_and_output_size_known_answers():
    # the tables of tests/poplin/RangeTest.cpp:33-168
    lib = capi.lib()
    for (stride, lo, hi), rows in RANGE_TABLE.items():
        p = capi.ConvParams.make(1, [10, 10], [3, 3], 1, 1, in_pad_lo=lo, in_pad_hi=hi, stride=stride)
        for out, k, expected in rows:
            assert lib.plb_conv_input_index(C.byref(p), 0, out, k) == expected
    for field, kernel, stride, lo, hi, expected in OUTPUT_DIM_TABLE:
        p = capi.ConvParams.make(1, list(field), list(kernel), 1, 1, in_pad_lo=list(lo),
                                 in_pad_hi=list(hi), stride=list(stride))
        assert tuple(p.output_field()) == expected


def test_geometry_matches_oracle_on_random_params():
    r = np.random.default_rng(3)
    lib, olib = capi.lib(), oracle._lib()
    for _ in range(200):
        spec = random_spec(r)
        p = _params_from_spec(spec)
        assert p.output_field() == spec.out_field()
        assert p.macs() == spec.macs()
        op = spec.to_c()
        for d, (o, k) in enumerate(zip(spec.out_field(), spec.kernel)):
            for oi in range(o):
                for ki in range(k):
                    assert lib.plb_conv_input_index(C.byref(p), d, oi, ki) == \
                        olib.oracle_conv_input_index(C.byref(op), d, oi, ki)


def test_flop_counts_of_the_benchmark_layers():
    mk = capi.ConvParams.make
    assert 2 * mk(32, [56, 56], [3, 3], 64, 64, padding=1).macs() == 7223640064
    assert 2 * mk(256, [28, 28], [3, 3], 128, 128, padding=1).macs() == 56405000192
    assert 2 * mk(256, [56, 56], [1, 1], 256, 512, stride=2).macs() == 52613349376
    assert 2 * mk(256, [224, 224], [7, 7], 3, 64, padding=3, stride=2).macs() == 59501838336  # 2*256*3*64*778^2


def test_validate_messages():
    # lib/poplin/ConvParams.cpp:172-266
    lib = capi.lib()

    def err(**kw):
        p = capi.ConvParams.make(1, [4, 4], [3, 3], 1, 1, **kw)
        rc = lib.plb_conv_validate(C.byref(p))
        return rc, lib.plb_last_error().decode()

    assert err()[0] == 0
    rc, msg = err(stride=[0, 1])
    assert rc == 1 and msg == "Stride must be non zero"
    rc, msg = err(in_dilation=[1, 0])
    assert rc == 1 and msg.startswith("Input dilation must be non zero")
    rc, msg = err(k_dilation=[0, 1])
    assert rc == 1 and msg.startswith("Kernel dilation must be non zero")
    rc, msg = err(in_trunc_lo=[3, 0], in_trunc_hi=[2, 0])
    assert rc == 1 and "truncates by more than the size of the field (4)" in msg
    rc, msg = err(k_trunc_lo=[2, 0], k_trunc_hi=[2, 0])
    assert rc == 1 and "truncates by more than the size of the kernel (3)" in msg
    rc, msg = err(k_trunc_lo=[3, 0])
    assert rc == 1 and msg == "Transformed kernel for dimension 0 has zero size"
    rc, msg = err(k_dilation=[2, 1])
    assert rc == 1 and msg == ("Transformed input size for dimension 0 (4) is less than the "
                               "transformed kernel size (5)")
    rc, msg = err(out_trunc_lo=[2, 0], out_trunc_hi=[1, 0])
    assert rc == 1 and "truncates by more than the size of the convolution output (2)" in msg


def test_planner_choices():
    plan = capi.conv_plan(capi.ConvParams.make(32, [56, 56], [3, 3], 64, 64, padding=1))
    assert (plan.tile_m, plan.tile_n) == (128, 64)
    assert plan.box_w * plan.box_h * plan.box_n == 128
    assert plan.tiles == 784 and plan.grid == 148          # no padded pixels
    assert plan.flops == 7223640064 and plan.bytes == 25763840
    plan = capi.conv_plan(capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1))
    assert plan.tile_n == 128 and plan.tiles == 1568
    plan = capi.conv_plan(capi.ConvParams.make(256, [56, 56], [1, 1], 256, 512, stride=2))
    assert plan.tile_n == 256 and plan.bytes == 308543488
    plan = capi.matmul_plan(capi.MatmulDesc.make(8192, 8192, 8192))
    assert plan.tile_n == 256 and plan.tiles == 2048 and plan.b_mn_major == 1
    assert plan.flops == 2 * 8192 ** 3 and plan.bytes == 3 * 8192 * 8192 * 2
    plan = capi.matmul_plan(capi.MatmulDesc.make(8192, 8192, 8192, input_type=capi.QUARTER))
    assert plan.bytes == 2 * 8192 * 8192 + 8192 * 8192 * 2
    plan = capi.matmul_plan(capi.MatmulDesc.make(5, 0, 4))
    assert plan.tiles == 0 and plan.flops == 0


def test_planner_rules_for_pairs_halo_tiles_and_padding():
    """What the closed-form planner picks, per layer shape (no GPU involved)."""
    c2 = capi.conv_plan(capi.ConvParams.make(32, [56, 56], [3, 3], 64, 64, padding=1))
    # small filter, one N tile: weights resident, one strip per filter column, CTA pairs
    assert (c2.resident_weights, c2.halo_rows, c2.cta_pair) == (1, 2, 1)
    c4 = capi.conv_plan(capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1))
    # weights too large to keep resident: streamed, but still one activation strip per column
    assert (c4.resident_weights, c4.halo_rows, c4.cta_pair) == (0, 2, 1)
    assert c4.box_w * c4.box_n % 8 == 0 and c4.stages >= 3
    bwd = capi.conv_plan(capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1), capi.PASS_TRAINING_BWD)
    assert bwd.b_mn_major == 1 and bwd.cta_pair == 1
    # a short K loop (4 steps) pairs only under 256-column tiles, where the weight tile is
    # most of a stage; with narrower tiles the lockstep costs more than it saves
    c3b = capi.conv_plan(capi.ConvParams.make(256, [56, 56], [1, 1], 256, 512, stride=2))
    assert (c3b.tile_n, c3b.cta_pair, c3b.halo_rows) == (256, 1, 0)
    short128 = capi.conv_plan(capi.ConvParams.make(256, [28, 28], [1, 1], 256, 128))
    assert (short128.tile_n, short128.cta_pair) == (128, 0)
    # a grid of a few tiles takes narrow tiles and no pairs
    c1 = capi.matmul_plan(capi.MatmulDesc.make(512, 1024, 1024))
    assert (c1.tile_n, c1.tiles, c1.grid, c1.cta_pair) == (64, 64, 64, 0)
    big = capi.matmul_plan(capi.MatmulDesc.make(8192, 8192, 8192))
    assert (big.tile_n, big.cta_pair, big.grid) == (256, 1, 148)
    # plan flags
    p = capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1)
    off = capi.conv_plan(p, capi.PASS_TRAINING_FWD, capi.ConvOptions.make(plan_flags=capi.PLAN_NO_CTA_PAIR | capi.PLAN_NO_HALO))
    assert (off.cta_pair, off.halo_rows) == (0, 0)
    small = capi.ConvParams.make(2, [12, 12], [3, 3], 64, 64, padding=1)
    assert capi.conv_plan(small).cta_pair == 0
    forced = capi.conv_plan(small, capi.PASS_TRAINING_FWD, capi.ConvOptions.make(plan_flags=capi.PLAN_FORCE_CTA_PAIR))
    assert forced.cta_pair == 1 and forced.grid % 2 == 0
    # channel counts that TMA cannot address are planned on their padded sizes
    odd = capi.conv_plan(capi.ConvParams.make(4, [9, 9], [3, 3], 20, 12, padding=1, groups=2))
    assert odd.tile_n == 64 and odd.tiles > 0
    assert capi.conv_plan(capi.ConvParams.make(4, [9, 9], [3, 3], 20, 12, padding=1), capi.PASS_TRAINING_BWD).tiles > 0
    # the stem goes to the small-channel path
    assert capi.conv_plan(capi.ConvParams.make(8, [224, 224], [7, 7], 3, 64, padding=3, stride=2)).kernel == 2
    # weight update: one strip per filter column with a unit vertical stride, K split to fill the device
    wu = capi.conv_wu_plan(capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1))
    assert (wu.kernel, wu.halo_rows, wu.tile_n, wu.split_k, wu.grid) == (1, 2, 384, 49, 147)
    # ... and tap groups sized so that two pipeline stages fit in shared memory
    wide = capi.conv_wu_plan(capi.ConvParams.make(4, [9, 13], [4, 4], 8, 24, stride=3))
    assert wide.halo_rows == 0 and wide.tile_n <= 10 * 32 and wide.stages >= 2


def test_pairs_of_wide_tiles_from_a_wave_on():
    """More than a wave (148) of tiles of 128 columns is paired whatever the stride and the groups."""
    for batch, side, chans, kw, paired in ((32, 56, 128, dict(stride=2), True), (12, 56, 256, dict(stride=2), True),
                                           (12, 28, 128, dict(groups=2), True), (5, 59, 392, dict(stride=2), True),
                                           (2, 59, 392, dict(stride=2), False), (32, 40, 128, dict(stride=2), False)):
        plan = capi.conv_plan(capi.ConvParams.make(batch, [side, side], [3, 3], chans, chans, padding=1, **kw))
        assert (plan.tiles > 148, plan.cta_pair, plan.split_k) == (paired, paired, 1)


def test_pairs_are_split_only_where_single_tiles_are():
    """A layer or product that runs whole on single SMs needs no scratch for pairs either."""
    mk = capi.ConvParams.make
    plan = lambda p, flags=0: capi.conv_plan(p, capi.PASS_TRAINING_FWD, capi.ConvOptions.make(plan_flags=flags))
    # more pairs than half the pair slots (74 on 148 SMs)
    for p in (mk(11, [16, 16], [5, 5], 304, 368, padding=2), mk(14, [15, 15], [5, 5], 248, 248, padding=2),
              mk(29, [19, 19], [3, 3], 504, 80, padding=1)):
        got = plan(p)
        assert (got.cta_pair, got.split_k, got.workspace_bytes) == (1, 1, 0)
    # a long reduction on few tiles
    few = plan(mk(1, [28, 28], [3, 3], 512, 512, padding=1))
    assert (few.cta_pair, few.split_k) == (1, 5)
    long = capi.matmul_plan(capi.MatmulDesc.make(488, 4312, 3992, transpose_b=True))
    assert (long.cta_pair, long.split_k, long.workspace_bytes) == (1, 1, 0)
    r = np.random.default_rng(7)
    split = 0
    for _ in range(400):
        chans_in, chans_out = (8 * int(r.integers(4, 64)) for _ in range(2))
        field = [int(r.integers(7, 60)) for _ in range(2)]
        kernel = int(r.choice([3, 5]))
        p = mk(int(r.integers(1, 16)), field, [kernel] * 2, chans_in, chans_out, padding=kernel // 2)
        got, single = plan(p), plan(p, capi.PLAN_NO_CTA_PAIR)
        if got.cta_pair:
            assert got.split_k == 1 or single.split_k > 1
            assert got.workspace_bytes == 0 or single.workspace_bytes > 0
            split += got.split_k > 1
    assert split > 0


def test_forced_resident_weights_with_splits_and_groups():
    """Residency that is asked for is kept with a forced K split, and with any number of
    groups that run side by side; with groups only one of the two is possible."""
    def plan(groups, flags, split=0, kernel=(3, 3), chans=64):
        p = capi.ConvParams.make(2, [12, 12], list(kernel), chans, chans, groups=groups, padding=1)
        f = capi.conv_plan(p, capi.PASS_TRAINING_FWD, capi.ConvOptions.make(plan_flags=flags, split_k=split))
        return f.resident_weights, f.split_k
    forced, pair = capi.PLAN_FORCE_RESIDENT_WEIGHTS, capi.PLAN_FORCE_CTA_PAIR
    for flags in (forced, forced | pair, forced | capi.PLAN_NO_HALO):
        assert plan(1, flags, split=3) == (1, 3)
        assert plan(3, flags, split=3) == (0, 3)
        assert plan(3, flags) == (1, 1) and plan(40, flags) == (1, 1)
    # 74 pairs or 148 CTAs run side by side
    assert plan(100, forced | pair) == (0, 1) and plan(100, forced | capi.PLAN_NO_CTA_PAIR) == (1, 1)
    assert plan(3, 0) == (0, 1)


def test_weight_update_plans_describe_what_runs():
    mk = capi.ConvParams.make
    # a first layer contracts windows of 64 over the rearranged input (4 x 16 channels of
    # 115 x 115 pixels), its 4 folded filter rows in one unit split over the device
    stem = capi.conv_wu_plan(mk(256, [224, 224], [7, 7], 3, 64, padding=3, stride=2))
    rearranged = (256 * 115 * 115 * 16 + 64) * 2
    assert (stem.split_k, stem.grid, stem.tile_n) == (148, 148, 4 * 64)
    assert stem.workspace_bytes == 148 * 4 * 64 * 64 * 4 + rearranged + 256
    # whole layers need the partial sums only, others copies of whole 128-byte rows too
    whole = capi.conv_wu_plan(mk(4, [9, 9], [3, 3], 64, 64, padding=1))
    assert whole.workspace_bytes == whole.split_k * 9 * 64 * 64 * 4
    ragged = capi.conv_wu_plan(mk(4, [9, 9], [3, 3], 20, 36, padding=1))
    pixels = 4 * 9 * 9
    assert ragged.workspace_bytes >= ragged.split_k * 9 * 20 * 36 * 4 + pixels * (64 + 128)
    # float: three planes of each operand
    pieces = capi.conv_wu_plan(mk(4, [9, 9], [3, 3], 64, 64, padding=1, input_type=capi.FLOAT, output_type=capi.FLOAT))
    assert pieces.workspace_bytes == pieces.split_k * 9 * 64 * 64 * 4 + 2 * 3 * ((pixels * 128 + 255) // 256 * 256)
    assert pieces.flops == whole.flops
    assert capi.conv_wu_plan(mk(4, [9, 9], [3, 3], 0, 64, padding=1)).tiles == 0


@pytest.mark.parametrize("n,field,kernel,ci,co,groups", [
    (39, [27, 7], [3, 1], 160, 64, 1), (30, [11, 7], [5, 2], 96, 60, 1), (7, [17, 37], [5, 1], 96, 64, 1),
    (1, [29, 57], [7, 1], 8, 32, 2), (64, [64, 64], [2, 1], 64, 64, 1), (2, [25, 88], [7, 1], 16, 32, 2), (256, [56, 56], [3, 3], 64, 64, 1)])
def test_saved_plans_of_weight_updates_reproduce_them(n, field, kernel, ci, co, groups):
    """A plan's split and strips given as constraints lead to the same tiling, where the tiles are
    fewer than the CTAs that there is room for, too."""
    p = capi.ConvParams.make(n, field, kernel, ci, co, groups=groups, padding=[k // 2 for k in kernel])
    free = capi.conv_wu_plan(p)
    fixed = capi.conv_wu_plan(p, capi.ConvOptions.make(split_k=free.split_k, plan_flags=0 if free.halo_rows or free.tile_m == 64 else capi.PLAN_NO_HALO))
    assert bytes(free) == bytes(fixed)


@pytest.mark.parametrize("rows,dilation,halo", [(2, 1, 0), (3, 1, 1), (4, 2, 2), (7, 1, 3)])
def test_halved_weight_updates_say_how_many_more_rows_they_read(rows, dilation, halo):
    """64 output channels' sums of all filter rows, from strips for one half of the filter rows."""
    plan = capi.conv_wu_plan(capi.ConvParams.make(64, [64, 64], [rows, 1], 64, 64, k_dilation=[dilation, 1]))
    assert (plan.tile_m, plan.tile_n, plan.halo_rows) == (64, rows * 64, halo)


@pytest.mark.parametrize("groups,chans,n,field,k", [(2, 8, 256, [56, 56], 3), (32, 8, 32, [28, 28], 3), (8, 8, 64, [40, 40], 5), (4, 16, 4, [9, 8], 3)])
def test_weight_update_plans_of_narrow_groups_describe_what_runs(groups, chans, n, field, k):
    """The shares of the pixels, whose partial sums are workspace; not the tensor-core route's, which
    constraints lead to."""
    p = capi.ConvParams.make(n, field, [k, k], chans, chans, groups=groups, padding=k // 2)
    plan = capi.conv_wu_plan(p)
    assert (plan.kernel, plan.in_place, plan.halo_rows) == (3, 0, k - 1)
    assert plan.workspace_bytes == plan.split_k * groups * k * k * chans * chans * 4
    assert plan.tiles == (groups * chans + 63) // 64 and plan.grid == plan.tiles * plan.split_k
    tiles = -(-field[1] // plan.box_w) * -(-field[0] // plan.box_h) * -(-n // plan.box_n)
    assert 1 <= plan.split_k <= tiles and plan.grid <= 148 * 3
    general = capi.conv_wu_plan(p, capi.ConvOptions.make(split_k=2))
    assert (general.kernel, general.split_k) == (1, 2) and general.flops == plan.flops


def test_plans_describe_the_operands_that_are_read():
    """Copies, pieces of floats and block-diagonal weights count as workspace; rows that are read
    where they lie are planned with their own pitch."""
    mk, r256 = capi.ConvParams.make, lambda n: (n + 255) // 256 * 256
    float_t = dict(input_type=capi.FLOAT, output_type=capi.FLOAT)
    # 56 channels are read in place: rows at odd multiples of 16 bytes, a long reduction is split
    flags = capi.PLAN_FORCE_CTA_PAIR | capi.PLAN_NO_RESIDENT_WEIGHTS | capi.PLAN_NO_HALO
    plan = capi.conv_plan(mk(2, [12, 12], [3, 8], 56, 56, padding=1), capi.PASS_TRAINING_FWD,
                          capi.ConvOptions.make(plan_flags=flags))
    assert plan.split_k > 1 and plan.workspace_bytes == plan.split_k * 2 * 12 * 7 * 64 * 4
    # with resident weights groups are not split
    plan = capi.conv_plan(mk(2, [12, 12], [3, 8], 56, 56, groups=3, padding=1), capi.PASS_TRAINING_FWD, capi.ConvOptions.make(
        plan_flags=capi.PLAN_FORCE_RESIDENT_WEIGHTS | capi.PLAN_FORCE_CTA_PAIR | capi.PLAN_NO_HALO))
    assert (plan.resident_weights, plan.split_k) == (1, 1)
    # 32 groups of 8: blocks of neighbouring groups, the same ones in both directions
    for kw, split in (({}, False), (float_t, True)):
        p = mk(4, [9, 9], [3, 3], 8, 8, groups=32, padding=1, **kw)
        fwd, bwd = capi.conv_plan(p, capi.PASS_TRAINING_FWD), capi.conv_plan(p, capi.PASS_TRAINING_BWD)
        assert fwd.tiles == bwd.tiles and fwd.tiles < 32 * 3
        assert fwd.workspace_bytes > 32 * 9 * 8 * 8 * (4 if split else 2) * 4
    # ragged rows: 40 bytes as 64; 3 pieces of 11 floats as 128 bytes; 33 quarters as 64
    ragged = capi.conv_plan(mk(4, [9, 9], [3, 3], 20, 36, padding=1))
    assert ragged.split_k == 1 and ragged.workspace_bytes == r256(4 * 81 * 64) + r256(9 * 36 * 64)
    floats = capi.matmul_plan(capi.MatmulDesc.make(100, 11, 50, transpose_b=True, **float_t))
    assert floats.workspace_bytes == r256(100 * 128) + r256(50 * 128)
    quarter = capi.matmul_plan(capi.MatmulDesc.make(100, 33, 50, input_type=capi.QUARTER, transpose_a=True))
    assert quarter.workspace_bytes == r256(100 * 64) + 50 * 64
    assert capi.matmul_plan(capi.MatmulDesc.make(512, 1024, 1024)).workspace_bytes == 0


@pytest.mark.parametrize("t", [capi.HALF, capi.FLOAT, capi.QUARTER])
def test_gradients_that_no_tap_reaches_are_cleared(t):
    """Input gradients of strided layers whose filter meets padding alone: there is no product
    for a kernel to form."""
    kw = dict(groups=4, input_type=t, output_type=capi.FLOAT if t == capi.FLOAT else capi.HALF, stride=2)
    for p in (capi.ConvParams.make(2, [1, 1], [1, 1], 8, 8, padding=1, **kw),
              capi.ConvParams.make(2, [1, 9], [1, 3], 8, 8, in_pad_lo=[1, 1], in_pad_hi=[1, 1], **kw)):
        assert capi.conv_plan(p, capi.PASS_TRAINING_BWD).kernel == 0


def test_plans_say_which_calls_read_their_operands_in_place():
    """One launch without workspace: few input channels, narrow groups, small products; not under
    constraints, whose tiling the plan holds."""
    mk, opt = capi.ConvParams.make, capi.ConvOptions.make
    route = lambda p, pass_=capi.PASS_TRAINING_FWD, o=None: (lambda q: (q.kernel, q.in_place))(capi.conv_plan(p, pass_, o))
    first = mk(256, [224, 224], [7, 7], 3, 64, padding=3, stride=2)
    assert route(first) == (2, 1) and capi.conv_plan(first).tile_n == 64
    for o in (opt(tile_n=64), opt(plan_flags=capi.PLAN_NO_HALO)):
        assert route(first, o=o) == (2, 0)
    assert route(mk(256, [224, 224], [7, 7], 3, 64, padding=3, stride=2, output_type=capi.FLOAT)) == (2, 0)
    # few channels in, and not 16 out
    assert route(mk(1, [9, 9], [1, 1], 1, 4)) == (3, 1) and route(mk(64, [30, 30], [3, 3], 2, 24, padding=1)) == (2, 0)
    groups = mk(2, [8, 13], [3, 3], 8, 8, groups=32, padding=1, stride=2)
    assert route(groups) == route(groups, capi.PASS_TRAINING_BWD) == (3, 1)
    assert route(groups, o=opt(split_k=1)) == (0, 0)
    wide = mk(256, [28, 28], [3, 3], 128, 128, padding=1)
    assert route(wide) == route(wide, capi.PASS_TRAINING_BWD) == (0, 0)
    products = [capi.matmul_plan(capi.MatmulDesc.make(*s)) for s in ((16, 512, 512), (8192, 8192, 8192))]
    assert [(q.kernel, q.in_place) for q in products] == [(3, 1), (0, 0)]


def test_products_of_impossible_pitches_keep_the_general_route():
    """Negative leading dimensions, and those beyond a tensor map's, are refused there."""
    for t, transpose_b, fields in ((capi.HALF, True, ("lda", "ldb")), (capi.HALF, False, ("lda", "ldb")),
                                   (capi.QUARTER, False, ("lda",))):
        for field in fields:
            for pitch, kernel in ((0, 3), (272, 3), (-256, 0), (2 ** 39, 0)):
                d = capi.MatmulDesc.make(16, 256, 128, input_type=t, transpose_b=transpose_b)
                setattr(d, field, pitch)
                assert capi.matmul_plan(d).kernel == kernel


def test_fused_all_reduce_needs_no_flags_for_layers_it_refuses():
    flags = lambda t: capi.lib().plb_conv_wu_allreduce_flag_bytes(
        C.byref(capi.ConvParams.make(4, [9, 9], [3, 3], 64, 64, padding=1, input_type=t, output_type=t)))
    assert flags(capi.HALF) > 0 and flags(capi.FLOAT) == 0


def test_3d_layers_plan_as_2d_layers_with_depth_folded_into_channels():
    """A 3-D field runs as the 2-D problem over the inner dimensions with the
    kernel depth folded into the channels: batch * out-depth images and KD * Ci
    input channels (forward, weight update), batch * depth images and KD * Co
    output channels (backward).  Planning also cross-checks the device-side depth
    index arithmetic against getInputIndex for every (output, kernel) pair."""
    p3 = capi.ConvParams.make(4, [6, 14, 14], [3, 3, 3], 64, 128, padding=1, stride=[2, 1, 1])
    od = p3.output_field()[0]
    assert od == 3
    fwd2 = capi.ConvParams.make(4 * od, [14, 14], [3, 3], 3 * 64, 128, padding=1)
    bwd2 = capi.ConvParams.make(4 * 6, [14, 14], [3, 3], 64, 3 * 128, padding=1)
    same = ("kernel", "tile_m", "tile_n", "stages", "grid", "tiles", "halo_rows", "cta_pair", "split_k")
    for pass_id, p2 in ((capi.PASS_TRAINING_FWD, fwd2), (capi.PASS_TRAINING_BWD, bwd2), (capi.PASS_TRAINING_WU, fwd2)):
        a, b = capi.conv_plan(p3, pass_id).as_dict(), capi.conv_plan(p2, pass_id).as_dict()
        assert {k: a[k] for k in same} == {k: b[k] for k in same}, pass_id
        assert a["flops"] == 2 * p3.macs()
    # every depth transform is accepted (it only changes the gather)
    odd = capi.ConvParams.make(2, [7, 5, 6], [3, 1, 3], 8, 16, in_pad_lo=[2, 0, 1], in_pad_hi=[0, 0, 1],
                               k_dilation=[2, 1, 1], in_dilation=[2, 1, 1], in_trunc_lo=[1, 0, 0],
                               k_flip=[1, 0, 0], in_flip=[1, 0, 0], out_pad_lo=[1, 0, 0], out_trunc_hi=[1, 0, 0],
                               stride=[2, 1, 1])
    for pass_id in (capi.PASS_TRAINING_FWD, capi.PASS_TRAINING_BWD, capi.PASS_TRAINING_WU):
        assert capi.conv_plan(odd, pass_id).flops == 2 * odd.macs()
    # input dilation in an inner dimension runs on the zero-stuffed input (2-D path's fallback)
    inner = capi.ConvParams.make(1, [4, 6, 6], [1, 3, 3], 16, 16, in_dilation=[1, 2, 1])
    stuffed = capi.ConvParams.make(4, [11, 6], [3, 3], 16, 16)
    assert capi.conv_plan(inner).tiles == capi.conv_plan(stuffed).tiles


def test_option_and_type_errors():
    with pytest.raises(capi.PlbError) as e:
        capi.matmul_plan(capi.MatmulDesc.make(4, 4, 4, input_type=capi.QUARTER, output_type=capi.FLOAT))
    assert e.value.code == 1 and "Output type must be half when input type is quarter" in e.value.message
    with pytest.raises(capi.PlbError) as e:
        capi.matmul_plan(capi.MatmulDesc.make(4, 4, 4, partials_type=capi.QUARTER))
    assert e.value.code == 2
    with pytest.raises(capi.PlbError) as e:
        capi.conv_plan(capi.ConvParams.make(1, [4, 4], [3, 3], 8, 8), opt=capi.ConvOptions.make(tile_n=96))
    assert e.value.code == 2


def _closed_context():
    """A context whose handle is null: every call gets as far as the library's own check."""
    ctx = capi.Context.__new__(capi.Context)
    ctx._h, ctx._ctx = C.c_void_p(), 0
    return ctx


def _per_layer_calls(ctx, desc, p, o):
    x = np.zeros(64, np.float32)
    return {
        "matmul": lambda: ctx.matmul(desc, x, x, None, x),
        "conv_fwd": lambda: ctx.conv_fwd(p, x, x, x, bias=None, opt=o),
        "convolution": lambda: ctx.convolution(p, x, x, x, x, o, True),
        "conv_bwd": lambda: ctx.conv_bwd(p, x, x, x, o),
        "conv_wu": lambda: ctx.conv_wu(p, x, x, None, x, o),
        "scaled_add_to": lambda: ctx.scaled_add_to(capi.HALF, x, x, 0.5, 8),
        "conv_bias_update": lambda: ctx.conv_bias_update(capi.HALF, x, 2, 4, capi.FLOAT, x, 0.5),
        "norm_moments": lambda: ctx.norm_moments(capi.HALF, x, 2, 4, 0.5, None, x, x),
        "norm_statistics": lambda: ctx.norm_statistics(capi.HALF, x, 2, 4, 1e-3, 1.0, x, x),
        "norm_normalise": lambda: ctx.norm_normalise(capi.HALF, x, x, x, x, x, 2, 4, None, x),
        "norm_whiten": lambda: ctx.norm_whiten(capi.HALF, x, x, x, 2, 4, x),
        "norm_scale_shift": lambda: ctx.norm_scale_shift(capi.HALF, x, x, None, 2, 4, x),
        "norm_param_gradients": lambda: ctx.norm_param_gradients(capi.HALF, x, x, 2, 4, 1.0, x, x),
        "norm_statistics_gradients": lambda: ctx.norm_statistics_gradients(capi.HALF, x, x, x, 2, 4, x),
        "cast_from_f32": lambda: ctx.cast_from_f32(capi.HALF, x, x, 8),
    }


@pytest.mark.parametrize("route", ["binding", "ctypes"])
def test_per_layer_calls_and_their_errors_by_either_route(monkeypatch, route):
    """The CPython binding and ctypes reach the same entry points and refuse the same arguments."""
    capi.lib()
    if route == "ctypes":
        monkeypatch.setattr(capi, "_BINDING", None)
    elif capi._BINDING is None:
        pytest.skip("the binding was not built")
    ctx, desc, p = _closed_context(), capi.MatmulDesc.make(4, 4, 4), capi.ConvParams.make(1, [4, 4], [3, 3], 8, 8)
    for o in (None, capi.ConvOptions.make()):
        for name, call in _per_layer_calls(ctx, desc, p, o).items():
            with pytest.raises(capi.PlbError) as e:
                call()
            assert "null context" in e.value.message, name
    # another structure, or bytes, in a descriptor's place
    for desc2, p2, o2 in ((p, desc, None), (bytes(4096), bytes(4096), None), (None, None, None), (p, p, p)):
        calls = _per_layer_calls(ctx, desc2, p2, o2)
        for name in ("conv_fwd", "convolution", "conv_bwd", "conv_wu") + (("matmul",) if o2 is None else ()):
            with pytest.raises((C.ArgumentError, TypeError)):
                calls[name]()
    for bad in (lambda: ctx.scaled_add_to("half", p, p, 0.5, 8), lambda: ctx.scaled_add_to(capi.HALF, None, None, 0.5, 8.0),
                lambda: ctx.scaled_add_to(capi.HALF, None, None, "half", 8)):
        with pytest.raises((C.ArgumentError, TypeError)):
            bad()
    if route == "binding":  # (ctypes cuts integers off)
        for bad in (lambda: ctx.norm_scale_shift(capi.HALF, None, None, None, 2, 2 ** 32 + 4, None),
                    lambda: ctx.cast_from_f32(2 ** 32 + capi.HALF, None, None, 8),
                    lambda: ctx.scaled_add_to(capi.HALF, None, None, 0.5, 2 ** 64)):
            with pytest.raises(OverflowError):
                bad()


def test_a_binding_that_cannot_be_used_is_passed_over(monkeypatch, tmp_path):
    """One that does not import is not used; one that cannot be built again does not stay."""
    import sys
    from poplibs_b200 import build
    capi.lib()
    monkeypatch.setattr(capi, "_BINDING", capi._BINDING)
    monkeypatch.setitem(sys.modules, "poplibs_b200._binding", None)  # importing it raises ImportError
    monkeypatch.delattr("poplibs_b200._binding", raising=False)
    capi._load_binding()
    assert capi._BINDING is None
    stale = tmp_path / "_binding.abi.so"
    untagged = tmp_path / "_binding.so"
    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setattr(build, "BINDING_OUT", str(stale))
    for why in ("no headers", "compile error"):
        stale.write_bytes(b""), untagged.write_bytes(b"")
        if why == "no headers":
            monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
        else:
            (tmp_path / "Python.h").write_text("#error not this one")
        assert build.build_binding(force=True) is None
        assert not stale.exists() and not untagged.exists()


def test_no_silent_fallback_without_a_gpu():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    with pytest.raises(capi.PlbError) as e:
        capi.Context(0)
    assert e.value.code == 4  # PLB_ERR_CUDA: fails loudly, nothing is computed on the host


def test_cpulist_parsing():
    """The kernel's cpulist format, as read from a PCI device's local_cpulist."""
    from poplibs_b200 import capi
    assert capi.parse_cpulist("0-3,8,10-11\n") == {0, 1, 2, 3, 8, 10, 11}
    assert capi.parse_cpulist("") == set()
    assert capi.parse_cpulist("5") == {5}

"""CPU-side checks of the boundary: the library loads and exports every symbol the
header declares, argument validation and plan selection behave, and the drop-in C++
names exist with the reference's mangling.  No kernel is launched."""
import ctypes
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol(pkg):
    header = open(os.path.join(ROOT, "include", "nmspmm_b200.h")).read()
    declared = set(re.findall(r"\b(nmspmm_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    lib = ctypes.CDLL(pkg.LIB_PATH)
    for name in sorted(declared):
        assert hasattr(lib, name), f"{name} declared in include/nmspmm_b200.h but not exported"
    assert declared == set(pkg.C_ABI_SYMBOLS)


def test_dropin_cpp_symbols_have_reference_mangling(pkg):
    """The reference's header declares C++ free functions (one takes int&), so the
    drop-in must export the same mangled names."""
    out = subprocess.run(["nm", "-D", "--defined-only", pkg.LIB_PATH], capture_output=True, text=True).stdout
    names = set(line.split()[-1] for line in out.splitlines() if line.strip())
    want = ["_Z26PreProcessing_low_sparsityPiiii", "_Z27PreProcessing_high_sparsityPiiiS_iiii", "_Z10transIndexPiiiiRiS0_"]
    for size in ("huge", "large", "medium", "small"):
        want.append(f"_Z{len('nmGEMM_' + size + '_matrices_low_sparsity')}nmGEMM_{size}_matrices_low_sparsityPfS_PiS_iiiifi")
        want.append(f"_Z{len('nmGEMM_' + size + '_matrices_high_sparsity')}nmGEMM_{size}_matrices_high_sparsityPfS_PiS0_S_iiiifi")
    for w in want:
        assert w in names, w


def test_status_strings(pkg):
    lib = pkg.load_library()
    assert lib.nmspmm_status_string(0) == b"ok"
    assert b"unsupported" in lib.nmspmm_status_string(pkg.UNSUPPORTED)
    assert lib.nmspmm_version() >= 0x000100


@pytest.mark.parametrize("M,N,K,n_keep,fmt,Ns,expect_tile", [
    (4096, 4096, 4096, 16, 0, 128, (128, 128)),
    (4096, 4096, 4096, 8, 1, 128, (128, 128)),
    (16, 11008, 4096, 8, 1, 128, (16, 128)),
    (64, 11008, 4096, 8, 1, 128, (64, 128)),
    (256, 11008, 4096, 8, 1, 128, (128, 128)),
    (192, 1024, 1024, 16, 0, 64, (64, 128)),
    (8192, 28672, 8192, 8, 1, 32, (128, 128)),
])
def test_plan_selection(pkg, M, N, K, n_keep, fmt, Ns, expect_tile):
    d = pkg.make_desc(M, N, K, n_keep, fmt, Ns)
    info = pkg.plan(d)
    assert (info.tile_m, info.tile_n) == expect_tile
    assert info.tiles_x == -(-N // info.tile_n) and info.tiles_y == -(-M // info.tile_m)
    ws = n_keep if fmt == 0 else 2 * n_keep
    n_win = K // 32 * n_keep // ws
    tiles = info.tiles_x * info.tiles_y
    assert info.stream_k == 1 and 1 <= info.n_virtual <= tiles * n_win
    assert info.grid == info.n_virtual and 0 <= info.n_dp <= tiles
    assert info.stages >= 2 and info.smem_bytes <= 227 * 1024
    need = pkg.workspace_bytes(d)
    assert need == 0 or need >= 2 * (info.n_virtual - info.n_dp) * info.tile_m * info.tile_n * 4


def _ranges(n_tiles, n_win, nv, n_dp):
    """Host restatement of the automatic unit schedule (virtual_range in gemm_args.h)."""
    out = [(v * n_win, (v + 1) * n_win) for v in range(n_dp)]
    base, total, n_sk = n_dp * n_win, (n_tiles - n_dp) * n_win, nv - n_dp
    out += [(base + i * total // n_sk, base + (i + 1) * total // n_sk) for i in range(n_sk)]
    return out


@pytest.mark.parametrize("n_tiles,n_win,nv,n_dp", [(1024, 64, 888 + 296, 888), (86, 64, 592, 0), (8, 2048, 296, 0),
                                                   (3, 5, 7, 0), (5, 1, 5, 0), (7, 3, 21, 0), (10, 4, 6 + 5, 6)])
def test_automatic_schedule_covers_every_unit_once(n_tiles, n_win, nv, n_dp):
    r = _ranges(n_tiles, n_win, nv, n_dp)
    assert r[0][0] == 0 and r[-1][1] == n_tiles * n_win and all(a[1] == b[0] for a, b in zip(r, r[1:]))
    total, n_sk = (n_tiles - n_dp) * n_win, nv - n_dp
    for t in range(n_tiles):
        holders = [v for v, (a, b) in enumerate(r) if a <= t * n_win + n_win - 1 and b > t * n_win]
        if t < n_dp:
            assert holders == [t]
        else:                                                   # tile_contributors() in gemm_args.h
            x0, x1 = (t - n_dp) * n_win, (t - n_dp) * n_win + n_win - 1
            v_first, v_last = n_dp + ((x0 + 1) * n_sk - 1) // total, n_dp + ((x1 + 1) * n_sk - 1) // total
            assert holders == list(range(v_first, v_last + 1))


def test_plan_balances_the_last_wave(pkg):
    info = pkg.plan(pkg.make_desc(2048, 3072, 4096, 8, 1, 128))               # 384 tiles: one full wave of 296 + 88
    tiles = info.tiles_x * info.tiles_y
    assert info.stream_k == 1 and 0 < info.n_dp < tiles and info.n_dp % (info.n_virtual - info.n_dp) == 0
    many = pkg.plan(pkg.make_desc(4096, 4096, 4096, 8, 1, 128))               # 1024 tiles: whole tiles only
    assert many.n_dp == many.n_virtual == 1024
    slab = pkg.plan(pkg.make_desc(8192, 3584, 8192, 8, 1, 128))                # 1792 tiles = 6 waves + 16 tiles: a nearly empty last wave is cut along k
    assert slab.n_dp == 6 * 296 and slab.n_virtual == 6 * 296 + 296
    exact = pkg.plan(pkg.make_desc(128 * 296 // 8, 1024, 4096, 8, 1, 128))      # 37 x 8 = 296 tiles: nothing to balance
    assert exact.n_dp == exact.tiles_x * exact.tiles_y == exact.n_virtual
    assert pkg.workspace_bytes(pkg.make_desc(128 * 296 // 8, 1024, 4096, 8, 1, 128)) == 0


def test_split_k_fills_the_machine_for_skinny_shapes(pkg):
    big = pkg.plan(pkg.make_desc(4096, 4096, 4096, 8, 1, 128))
    assert big.split_k == 1 and big.grid == big.n_virtual
    skinny = pkg.plan(pkg.make_desc(16, 11008, 4096, 8, 1, 128))
    assert skinny.split_k > 1 and skinny.n_virtual > 86
    deep = pkg.plan(pkg.make_desc(128, 1024, 131072, 4, 1, 128))
    assert deep.split_k >= 16
    forced = pkg.plan(pkg.make_desc(128, 1024, 131072, 4, 1, 128, split_k=7))
    assert forced.split_k == 7 and forced.stream_k == 0 and forced.n_virtual == 8 * 7
    clamped = pkg.plan(pkg.make_desc(128, 128, 64, 16, 0, 128, split_k=9))
    assert clamped.split_k == 2            # only two windows exist
    # the tensor-core path: slices when the tiles alone leave SMs idle, pieces always in scratch
    tdeep = pkg.make_desc(128, 1024, 131072, 4, 1, 128, path=pkg.PATH_TF32)
    info = pkg.plan(tdeep)
    assert info.tile_n == 256 and info.split_k == 148 // 4 and info.grid == 4 * info.split_k      # four wide tiles, one CTA per SM
    assert pkg.workspace_bytes(tdeep) == (64 << 10) + info.grid * 128 * 256 * 4      # counter block + one slot per slice
    # 512 tiles on 148 one-CTA SMs: three whole waves, the 68 tiles of the last one in two slices each
    tbig = pkg.plan(pkg.make_desc(4096, 4096, 4096, 8, 1, 128, path=pkg.PATH_TF32))
    assert tbig.tile_n == 256 and tbig.n_dp == 444 and tbig.split_k == 2 and tbig.grid == 444 + 2 * 68
    tlow = pkg.plan(pkg.make_desc(4096, 4096, 4096, 16, 0, 128, path=pkg.PATH_TF32))
    assert tlow.tile_n == 256 and tlow.n_dp == 444 and tlow.grid == 444 + 2 * 68   # the wide tile for every ratio once it fills the GPU
    tsmall = pkg.plan(pkg.make_desc(1024, 128, 4096, 16, 0, 128, path=pkg.PATH_TF32))
    assert tsmall.tile_n == 128                                                # B narrower than the wide tile
    texact = pkg.plan(pkg.make_desc(128 * 148, 256, 4096, 8, 1, 128, path=pkg.PATH_TF32))    # exactly one wave: nothing to slice
    assert texact.split_k == 1 and texact.grid == 148 and pkg.workspace_bytes(pkg.make_desc(128 * 148, 256, 4096, 8, 1, 128, path=pkg.PATH_TF32)) == 0
    one = pkg.plan(pkg.make_desc(128, 128, 64, 16, 0, 128, split_k=1))
    assert one.split_k == 1 and pkg.workspace_bytes(pkg.make_desc(128, 128, 64, 16, 0, 128, split_k=1)) == 0


@pytest.mark.parametrize("kw,status", [
    (dict(M=0), 1), (dict(N=100), 1), (dict(K=48), 1), (dict(M=6), 1), (dict(layout_ns=96), 1),
    (dict(n_keep=10), 2), (dict(n_keep=16, fmt=1), 2), (dict(n_keep=4, fmt=0), 2), (dict(path=2), 2), (dict(vec_len=48), 1), (dict(vec_len=64, N=160, layout_ns=32), 1),
    (dict(N=192, layout_ns=128), 1), (dict(K=96, n_keep=8, fmt=1), 1), (dict(split_k=-1), 1),
])
def test_bad_descriptions_are_rejected(pkg, kw, status):
    base = dict(M=128, N=256, K=256, n_keep=16, fmt=0, layout_ns=128, path=0, split_k=0, vec_len=0)
    base.update(kw)
    d = pkg.make_desc(base["M"], base["N"], base["K"], base["n_keep"], base["fmt"], base["layout_ns"],
                      base["path"], base["split_k"], 0, base["vec_len"])
    info = pkg.PlanInfo()
    rc = pkg.load_library().nmspmm_gemm_plan(ctypes.byref(d), ctypes.byref(info))
    assert rc == status, (kw, rc)


def test_sparsity_argument_mapping(pkg):
    assert [pkg.n_keep_of(s) for s in (0.0, 0.5, 0.625, 0.75, 0.875)] == [32, 16, 12, 8, 4]
    assert [pkg.format_of(n) for n in (32, 16, 12, 8, 4)] == [0, 0, 0, 1, 1]
    with pytest.raises(ValueError):
        pkg.n_keep_of(0.3)


def test_partition_columns(pkg_host):
    sh = pkg_host.sharding
    assert sh.partition_columns(28672, 8, 128) == [(i * 3584, (i + 1) * 3584) for i in range(8)]
    parts = sh.partition_columns(11008, 4, 128)          # 86 blocks over 4 ranks: 22, 22, 21, 21
    assert [c1 - c0 for c0, c1 in parts] == [2816, 2816, 2688, 2688]
    assert parts[0][0] == 0 and parts[-1][1] == 11008 and all(a[1] == b[0] for a, b in zip(parts, parts[1:]))
    with pytest.raises(ValueError):
        sh.partition_columns(256, 4, 128)
    with pytest.raises(ValueError):
        sh.partition_columns(200, 1, 128)


def test_tuned_plan_table_overrides_the_heuristics_and_only_them(pkg, tmp_path):
    d = pkg.make_desc(256, 2048, 2048, 4, 1, 128)
    base = pkg.plan(d)
    try:
        pkg.set_tuned_plan(d, 2, 4)                                    # tile 64 x 128, four K slices
        tuned = pkg.plan(d)
        assert (tuned.tile_m, tuned.tile_n, tuned.split_k) == (64, 128, 4)
        # a caller that names a tile or a split keeps its own choice
        own = pkg.plan(pkg.make_desc(256, 2048, 2048, 4, 1, 128, tile=1))
        assert (own.tile_m, own.tile_n) == (128, 128)
        assert pkg.plan(pkg.make_desc(256, 2048, 2048, 4, 1, 128, split_k=2)).split_k == 2
        # other shapes are untouched
        other = pkg.plan(pkg.make_desc(512, 2048, 2048, 4, 1, 128))
        assert (other.tile_m, other.tile_n) == (pkg.plan(pkg.make_desc(512, 2048, 2048, 4, 1, 128, tile=0)).tile_m, other.tile_n)
        # the file form
        table = tmp_path / "plans.txt"
        pkg.tuner.write_table(str(table), [((128, 1024, 4096, 8, 1, 0, 32), 3, 2, 1.0, 2.0), ((64, 256, 256, 16, 0, 0, 32), 0, 0, 1.0, 1.0)])
        assert pkg.tuner.read_table(str(table)) == {(128, 1024, 4096, 8, 1, 0, 32): (3, 2)}
        pkg.clear_tuned_plans()
        assert pkg.load_tuned_plans(str(table)) == 1
        got = pkg.plan(pkg.make_desc(128, 1024, 4096, 8, 1, 128))
        assert (got.tile_m, got.split_k) == (32, 2)
    finally:
        pkg.clear_tuned_plans()
    again = pkg.plan(d)
    assert (again.tile_m, again.tile_n, again.split_k) == (base.tile_m, base.tile_n, base.split_k)


def test_tf32_forms_are_selected_by_tile_id(pkg):
    """Tile ids 8 and 9 force the gathering and the expanding form of the TF32 path; the
    expanding one exists for the 32-k formats only and neither exists on the exact path."""
    low = pkg.make_desc(512, 1024, 1024, 16, pkg.FORMAT_LOW, 128, pkg.PATH_TF32)
    for tile, threads in ((pkg.TILE_128x256_GATHER, 256), (pkg.TILE_128x256_EXPAND, 320)):
        d = pkg.make_desc(512, 1024, 1024, 16, pkg.FORMAT_LOW, 128, pkg.PATH_TF32, 0, tile)
        info = pkg.plan(d)
        assert (info.tile_m, info.tile_n, info.threads) == (128, 256, threads)
    assert pkg.plan(low).tile in (pkg.TILE_128x256, pkg.TILE_128x256_EXPAND)
    assert pkg.plan(pkg.make_desc(512, 1024, 1024, 16, pkg.FORMAT_LOW, 128, pkg.PATH_TF32, 0, pkg.TILE_128x128)).tile == pkg.TILE_128x128
    lib = pkg.load_library()
    high = pkg.make_desc(512, 1024, 1024, 8, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32, 0, pkg.TILE_128x256_EXPAND)
    assert lib.nmspmm_gemm_workspace_bytes(ctypes.byref(high)) == 0
    with pytest.raises(pkg.NMSpMMError):
        pkg.plan(high)
    for tile in (pkg.TILE_128x256_GATHER, pkg.TILE_128x256_EXPAND):
        with pytest.raises(pkg.NMSpMMError):
            pkg.plan(pkg.make_desc(512, 1024, 1024, 16, pkg.FORMAT_LOW, 128, pkg.PATH_FP32, 0, tile))


def test_banded_tile_order_visits_every_tile_once(tmp_path):
    """gemm_args.h::tile_coords (shared by host and device): for plain and banded orders, full and
    ragged last bands, every (row, column) of tiles is produced by exactly one tile number, tiles
    of a band are consecutive, and band 0 is the row-by-row order."""
    src = tmp_path / "order.cpp"
    src.write_text(r'''
#include <cstdio>
#include <vector>
#include "gemm_args.h"
using namespace nmspmm;
int main() {
    const int shapes[][3] = {{5, 4, 0}, {5, 4, 2}, {112, 64, 16}, {7, 3, 3}, {8, 1, 4}, {9, 5, 127}, {33, 2, 8}, {224, 64, 32}};
    for (auto& sh : shapes) {
        const int tx_n = sh[0], ty_n = sh[1], band = sh[2];
        if (band >= tx_n && band != 0) continue;               // the planner never packs a band that wide
        const int packed = pack_tiles_x(tx_n, band);
        std::vector<int> seen(tx_n * ty_n, 0);
        int last_band = -1;
        for (int t = 0; t < tx_n * ty_n; ++t) {
            int ty, tx;
            tile_coords(t, packed, ty_n, ty, tx);
            if (ty < 0 || ty >= ty_n || tx < 0 || tx >= tx_n) { std::printf("range %d %d %d: tile %d -> %d %d\n", tx_n, ty_n, band, t, ty, tx); return 1; }
            if (seen[ty * tx_n + tx]++) { std::printf("twice %d %d %d: tile %d\n", tx_n, ty_n, band, t); return 1; }
            if (band == 0 && (ty != t / tx_n || tx != t % tx_n)) { std::printf("plain order broken at %d\n", t); return 1; }
            if (band > 0) {
                const int b = tx / band;
                if (b < last_band) { std::printf("band order %d %d %d: tile %d\n", tx_n, ty_n, band, t); return 1; }
                last_band = b;
            }
        }
    }
    std::printf("ok\n");
    return 0;
}
''')
    exe = tmp_path / "order"
    inc = os.path.join(ROOT, "nm-spmm_b200", "csrc")
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr


def test_few_rows_plans(pkg):
    """TF32 path, M <= 64: the library takes the 16 / 32 / 64-row tiles by itself, cuts K so that no
    slice has more windows than a CTA's index list holds, and refuses what the form cannot do."""
    for M, rows in ((1, 16), (16, 16), (17, 32), (32, 32), (33, 64), (64, 64)):
        info = pkg.plan(pkg.make_desc(M + (-M) % 4, 11008, 4096, 8, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32))
        assert (info.tile_m, info.tile_n, info.threads) == (rows, 128, 128)
        assert info.tiles_y == 1 and info.tiles_x == 86 and info.grid == 86 * info.split_k
        assert -(-64 // info.split_k) <= 24                       # windows per slice (K / 64 = 64 merged windows)
    assert pkg.plan(pkg.make_desc(68, 11008, 4096, 8, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32)).tile_m == 128
    deep = pkg.plan(pkg.make_desc(64, 1024, 131072, 4, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32))
    assert deep.tile_m == 64 and -(-2048 // deep.split_k) <= 24
    lib = pkg.load_library()
    too_few = pkg.make_desc(16, 1024, 131072, 4, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32, 2, pkg.TILE_16x128)
    assert lib.nmspmm_gemm_workspace_bytes(ctypes.byref(too_few)) == 0   # 1024 windows per slice: refused
    # left to the library, the same split goes to the 128-row tiles instead
    assert pkg.plan(pkg.make_desc(16, 1024, 131072, 4, pkg.FORMAT_HIGH, 128, pkg.PATH_TF32, 2)).tile_m == 128


def test_slices_of_equal_length_where_they_fill_the_slots(pkg):
    """The last partial wave is cut into whole slices per tile when those keep 95 % of the CTA slots busy
    (148 SMs), into ranges that cross tiles otherwise."""
    whole = pkg.plan(pkg.make_desc(776, 5760, 2048, 8, 1, 128))                # 13 x 45 = 585 of 592: one slice per tile
    assert (whole.tile_m, whole.n_dp, whole.n_virtual) == (64, 0, 585)
    assert pkg.workspace_bytes(pkg.make_desc(776, 5760, 2048, 8, 1, 128)) == 0
    assert pkg.plan(pkg.make_desc(1536, 1536, 8192, 8, 1, 128)).n_virtual == 288   # 144 tiles, two slices each
    ranges = pkg.plan(pkg.make_desc(256, 4096, 4096, 8, 1, 128))               # 64 tiles: four slices each would leave 40 of 296 idle
    assert ranges.n_virtual == 296


@pytest.mark.parametrize("M,N,K,n_keep,n_virtual", [
    (4, 12032, 2048, 12, 592), (4, 24960, 5120, 4, 592), (12, 24448, 1536, 4, 592), (20, 24704, 1536, 4, 592),   # rows of A not whole 64 bytes
    (16, 24320, 4096, 4, 570), (32, 14848, 1024, 12, 580), (64, 10752, 4096, 16, 588),     # little left idle
    (48, 12032, 22016, 16, 592), (192, 24064, 22016, 16, 592), (128, 6016, 14336, 16, 296), (256, 640, 120128, 8, 296)])  # too much left idle for too long
def test_slices_of_equal_length_only_where_they_pay(pkg, M, N, K, n_keep, n_virtual):
    """Plans of less than a wave whose equal slices would keep 95 % of the slots: taken where the idle share times
    the kept rows is at most 100, and on few-row tiles where M is a multiple of 16."""
    assert pkg.plan(pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128)).n_virtual == n_virtual


@pytest.mark.parametrize("M,K,n_keep,tile_m", [(192, 2080, 12, 64), (320, 2080, 12, 128), (776, 2080, 16, 128), (320, 480, 12, 64),
                                               (320, 2048, 8, 64), (192, 4096, 16, 64), (1032, 4096, 12, 128)])
def test_tile_of_the_exact_path_follows_padding_and_pairs(pkg, M, K, n_keep, tile_m):
    assert pkg.plan(pkg.make_desc(M, 4096, K, n_keep, pkg.format_of(n_keep), 128)).tile_m == tile_m


@pytest.mark.parametrize("M,N,K,n_keep,narrow", [(256, 11008, 4096, 16, True), (2048, 9472, 4096, 8, False), (1024, 640, 4096, 12, True),
                                                 (168, 1664, 8320, 12, False), (84, 512, 6976, 16, False), (96, 640, 9152, 4, False), (1248, 1920, 2496, 8, False)])
def test_calls_take_192_columns_where_they_are_faster(pkg, M, N, K, n_keep, narrow):
    d = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128, pkg.PATH_TF32)
    assert pkg.plan(d).tile == pkg.TILE_128x256
    assert pkg.call_plan(d).tile == (pkg.TILE_128x192 if narrow else pkg.TILE_128x256)


def test_what_rows_of_16_bits_take_is_asked_for(pkg):
    """Their steps have lengths of their own, so their plan may be another than that of FP32 rows or of a copy: what the
    entries ask for holds either."""
    lib, base, M = pkg.load_library(), 1 << 20, 256
    differ = 0
    for N in (640, 1024, 2560, 4096):
        for n_keep in (16, 12, 8, 4):
            d, K = ctypes.byref(pkg.make_desc(M, N, 2048, n_keep, pkg.format_of(n_keep), 128, pkg.PATH_TF32)), 2048
            far = base + 4 * M * K
            rows, copied = (lib.nmspmm_gemm_row_major_call_bytes(d, pkg.DTYPE_BF16, a, far) for a in (base, base + 2))
            differ += rows != copied - 4 * M * K
            assert lib.nmspmm_gemm_row_major_16_workspace_bytes(d) == max(rows + 4 * M * K, copied)
    assert differ


@pytest.mark.parametrize("M,N,K,n_keep", [(512, 24576, 8192, 4), (512, 24576, 8192, 8), (1024, 12288, 4096, 4), (1024, 12288, 4096, 8),
                                          (1024, 22016, 8192, 8), (2048, 6144, 2048, 8)])
def test_tuned_shapes_keep_an_entry_for_callers_with_the_named_scratch(pkg, M, N, K, n_keep):
    """These ran a tuned tile on the scratch of nmspmm_gemm_workspace_bytes before calls took wide tiles by themselves: without an
    entry that scratch is none, and a caller who sizes by it would be back on the untuned tile."""
    d = pkg.make_desc(M, N, K, n_keep, 1, 128)
    saved = pkg.tuned_plans_snapshot_and_clear()
    try:
        pkg.load_tuned_plans(pkg.tuner.default_table_path())
        assert pkg.plan(d).tile == pkg.call_plan(d, pkg.workspace_bytes(d)).tile == pkg.TILE_128x256
        assert pkg.tuner.tile_for_less_scratch(pkg, (M, N, K, n_keep, 1, 0, 32)) == pkg.TILE_128x256      # tuning keeps it
        assert pkg.tuner.tile_for_less_scratch(pkg, (256, 8192, 22016, 4, 1, 0, 32)) == 0                 # the named scratch is enough here
    finally:
        pkg.tuned_plans_restore(saved)


def test_the_few_rows_kernels_do_not_spill(pkg_host):
    """What ptxas said when the library was built: the 64-row tiles have 128 registers for four CTAs per SM."""
    report = os.path.join(pkg_host.build.OBJ, "gemm_tf32_few_rows.cu.o.ptxas.txt")
    if not os.path.exists(report):
        pytest.skip("built without ptxas' report")
    spills = [int(n) for n in re.findall(r"(\d+) bytes spill stores", open(report).read())]
    assert len(spills) >= 12 and not any(spills)


def test_counter_bytes_are_asked_for_only_by_plans_that_use_counters(pkg):
    def counters(*args):
        return pkg.load_library().nmspmm_gemm_counter_bytes(ctypes.byref(pkg.make_desc(*args)))
    assert counters(128, 256, 2048, 16, 0, 128, 0, 2) == 256             # two pieces per tile, added by the last to arrive
    assert counters(128, 256, 2048, 16, 0, 128, 0, 8) == 0               # eight: the reduction kernel
    assert counters(128, 256, 2048, 16, 0, 128, 0, 1) == 0               # whole tiles
    assert counters(3, 11008, 4096, 8, 1, 128, 1) == 0                   # TF32, any row count


def test_row_major_scratch_is_what_the_call_writes(pkg):
    """The tensor-core path reads rows and stores 16 bits itself: no FP32 copies of A or C are asked for, unless A
    is off a 16-byte boundary, C overlaps A, or the weight is unpruned."""
    lib, base = pkg.load_library(), 1 << 20
    M, N, K = 8192, 28672, 8192
    tf32 = ctypes.byref(pkg.make_desc(M, N, K, 8, 1, 128, pkg.PATH_TF32, 0, 0, 64))
    exact = ctypes.byref(pkg.make_desc(M, N, K, 8, 1, 128, pkg.PATH_FP32))
    dense = ctypes.byref(pkg.make_desc(M, N, K, 32, 0, 128, pkg.PATH_TF32))
    far, copy_a, copy_c = base + 4 * M * K, 4 * M * K, 4 * M * N

    def call(desc, dtype, a=base, c=far):
        return lib.nmspmm_gemm_row_major_call_bytes(desc, dtype, a, c)

    for dtype in (pkg.DTYPE_F32, pkg.DTYPE_F16, pkg.DTYPE_BF16):
        own = call(tf32, dtype)
        assert 0 < own < 32 << 20
        assert call(tf32, dtype, a=base + 8) == call(tf32, dtype, c=base + 4096) == own + copy_a
        assert call(exact, dtype) >= copy_a + (0 if dtype == pkg.DTYPE_F32 else copy_c)
    assert call(dense, pkg.DTYPE_F16) >= copy_a > call(dense, pkg.DTYPE_F32)
    assert lib.nmspmm_gemm_row_major_16_workspace_bytes(tf32) == own + copy_a       # whatever A is, without an FP32 C
    assert lib.nmspmm_gemm_row_major_workspace_bytes(tf32) == own + copy_a


@pytest.mark.parametrize("M,N,K,n_keep,tile", [
    (4096, 4096, 4096, 8, (128, 256)), (128, 1024, 131072, 4, (128, 256)), (64, 11008, 4096, 8, (64, 512)), (6512, 3200, 4096, 8, (256, 128)),
    (32, 11008, 4096, 8, None), (5440, 1792, 640, 8, None), (128, 512, 1024, 16, None), (4096, 4096, 4096, 32, None)])
def test_calls_take_a_wide_tile_where_it_pays_and_fits(pkg, M, N, K, n_keep, tile):
    """148 SMs: the tile a call runs with all the scratch it asks for, and what it runs with less."""
    d = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128)
    base, call = pkg.plan(d), pkg.call_plan(d)
    assert (call.tile_m, call.tile_n) == (tile or (base.tile_m, base.tile_n))
    need, more = pkg.workspace_bytes(d), pkg.call_workspace_bytes(d)
    assert more >= need
    own = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128, 0, 0, call.tile)
    for scratch in (0, need, more):                              # never a plan whose pieces do not fit
        ran = pkg.call_plan(d, scratch)
        assert ran.tile == base.tile or pkg.workspace_bytes(own) <= scratch
    for named in (dict(tile=1), dict(split_k=2)):                # the caller's tile or split stays
        e = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128, 0, named.get("split_k", 0), named.get("tile", 0))
        assert pkg.call_plan(e).tile == pkg.plan(e).tile
    try:
        pkg.set_tuned_plan(d, 2, 4)                              # so does a tuned entry
        assert pkg.call_plan(d).tile == pkg.TILE_64x128
    finally:
        pkg.clear_tuned_plans()


@pytest.mark.parametrize("M,N,K,n_keep,path", [(4096, 4096, 4096, 8, 0), (4096, 4096, 4096, 16, 0), (2048, 5760, 1024, 16, 0),
                                               (512, 11008, 1024, 12, 0), (132, 1024, 1024, 16, 1), (256, 1024, 1024, 12, 1)])
def test_a_row_major_call_takes_the_named_plans_scratch(pkg, M, N, K, n_keep, path):
    """Scratch for the plan that a description names, too little for the one a call prefers: planned all the same (the
    launch then fails for want of a GPU).  Before the preferred plan was cleared away its sizes stayed and the call was refused."""
    if pytest.importorskip("torch").cuda.is_available():
        pytest.skip("the operands are made-up addresses; test_gpu_wide_tiles.py runs such calls")
    d = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128, path)
    lib, ref, own = pkg.load_library(), ctypes.byref(d), pkg.workspace_bytes(d)
    assert own < pkg.call_workspace_bytes(d)
    copy_a = 0 if path == pkg.PATH_TF32 else 4 * M * K
    less = max(own, 64 << 10) + copy_a
    at = [ctypes.c_void_p((1 << 20) + (i << 32)) for i in range(6)]
    assert lib.nmspmm_gemm_row_major(ref, *at[:4], at[4], at[5], less, None) == pkg.CUDA_ERROR
    assert lib.nmspmm_gemm_row_major(ref, *at[:4], at[4], at[5], less - 1, None) == pkg.WORKSPACE_TOO_SMALL
    if path == pkg.PATH_TF32:
        assert lib.nmspmm_gemm_row_major_16(ref, pkg.DTYPE_BF16, *at[:4], at[4], at[5], less, None) == pkg.CUDA_ERROR

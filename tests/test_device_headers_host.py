"""The device headers compile for the host (their PTX wrappers have host stand-ins), which is how the CPU plumbing runs
the same protocol code.  Layout constants and helpers of the data-as-flag transport, and a send -> check -> receive
round trip of both packed formats on host memory.  (Reference: tests/data_as_flag/unit: 512 / 480 / 32 bytes,
flag at offset 480, eight floats of 1.0, block counts 0 -> 0, 480 -> 1, 481 -> 2.)"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r'''
#include <cstdio>
#include <cstring>
#include <vector>
#include "device/tilexr_data_as_flag.cuh"
using namespace tilexr;
static_assert(DATA_AS_FLAG_BLOCK_BYTES == 512 && DATA_AS_FLAG_PAYLOAD_BYTES == 480 && DATA_AS_FLAG_FLAG_BYTES == 32, "block");
static_assert(DATA_AS_FLAG_FLAG_OFFSET == 480 && DATA_AS_FLAG_FLAG_FLOATS == 8, "flag");
int main()
{
    if (DataAsFlagBlockCount(0) != 0 || DataAsFlagBlockCount(480) != 1 || DataAsFlagBlockCount(481) != 2) return 1;
    if (DataAsFlagPackedBytes(481) != 1024 || Ll16UnitCount(13) != 2 || Ll16PackedBytes(24) != 32) return 2;
    CommArgs args;
    std::memset(&args, 0, sizeof(args));
    args.extraFlag = TileXR::TILEXR_FLAG_HOST_MEMORY;
    args.waitTimeoutNs = 1000000;
    args.rankSize = 1;
    std::vector<unsigned char> window(TILEXR_WIN_DATA_OFFSET, 0);      // control block and flag planes of rank 0
    args.peerMems[0] = window.data();
    args.peerMemBytes = window.size();
    Waiter w = MakeWaiter(&args, 7, 0);
    const uint64_t n = 1008;                      // whole 16-byte vectors and 12-byte units, not whole 480-byte blocks
    auto nosync = [] {};
    std::vector<unsigned char> src(n + 16), packed(DataAsFlagPackedBytes(n) + 64, 0), out(n + 16, 0);
    for (uint64_t i = 0; i < n; ++i) src[i] = static_cast<unsigned char>(i * 7 + 3);
    if (DataAsFlagCheck(packed.data(), DataAsFlagBlockCount(n), w.epoch)) return 3;      // nothing has arrived yet
    DataAsFlagSend(packed.data(), src.data(), n, w.epoch, 0, 1, nosync);
    if (!DataAsFlagCheck(packed.data(), DataAsFlagBlockCount(n), w.epoch)) return 4;
    if (!DataAsFlagCheckAndRecv(w, out.data(), packed.data(), n, 0, 0, 1, nosync)) return 5;
    if (std::memcmp(out.data(), src.data(), n) != 0) return 6;
    std::vector<unsigned char> ll(Ll16PackedBytes(n) + 64, 0), out2(n + 16, 0);
    Ll16Send(ll.data(), src.data(), n, w.epoch, 0, 1);
    if (!Ll16Recv(w, out2.data(), ll.data(), n, 0, 0, 1)) return 7;
    if (std::memcmp(out2.data(), src.data(), n) != 0) return 8;
    // a batch that never arrives: the bounded wait gives up and says so
    std::vector<unsigned char> empty(Ll16PackedBytes(n) + 64, 0);
    Waiter w2 = MakeWaiter(&args, 9, 0);
    if (Ll16Recv(w2, out2.data(), empty.data(), n, 0, 0, 1)) return 9;
    if (w2.ok()) return 10;
    std::puts("ok");
    return 0;
}
'''


def test_data_as_flag_layout_and_round_trip_on_the_host(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "daf.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "daf"
    proc = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc' / 'include'}", str(src), "-o", str(exe)],
                          capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr[-3000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == "ok", (run.returncode, run.stdout, run.stderr)


UDMA_PROGRAM = r'''
#include <cstdio>
#include <cstring>
#include <vector>
#include "device/tilexr_udma.cuh"
using namespace tilexr;
int main()
{
    // two ranks whose registered regions live in this process; the program plays rank 0
    constexpr uint64_t BYTES = 4096;
    std::vector<unsigned char> region0(BYTES, 0), region1(BYTES, 0);
    uint8_t *peers[2] = {region0.data(), region1.data()};
    TileXR::TileXRRegistry reg;
    std::memset(&reg, 0, sizeof(reg));
    reg.magic = TILEXR_REGISTRY_MAGIC;
    reg.rankSize = 2;
    reg.regionCount = 1;
    reg.regions[0].bytes = BYTES;
    reg.regions[0].localBase = peers[0];
    reg.regions[0].peerBase = peers;
    CommArgs args;
    std::memset(&args, 0, sizeof(args));
    args.rank = 0;
    args.rankSize = 2;
    args.extraFlag = TileXR::TILEXR_FLAG_HOST_MEMORY;
    if (UDMAEnabled(&args) || UDMAQpCount(&args) != 0) return 1;                   // no registry, no verbs
    args.extraFlag |= TileXR::TILEXR_FLAG_RMA;
    args.registryPtr = &reg;
    if (!UDMAEnabled(&args) || !UDMARegistryEnabled(&args) || UDMAQpCount(&args) == 0) return 2;
    if (!UDMARankValid(&args, 1) || UDMARankValid(&args, 0) || UDMARankValid(&args, 2)) return 3;   // a peer, never itself
    std::vector<unsigned char> src(512), back(512, 0);
    for (size_t i = 0; i < src.size(); ++i) src[i] = static_cast<unsigned char>(i * 5 + 1);
    if (UDMAPutNbiOnQp<unsigned char>(&args, 1, 0, src.data(), 1024, 512) != TILEXR_UDMA_STATUS_SUCCESS) return 4;
    UDMAQuiet(&args, 1);
    if (std::memcmp(region1.data() + 1024, src.data(), 512) != 0) return 5;
    if (UDMAGetNbiOnQp<unsigned char>(&args, 1, 3, back.data(), 1024, 512) != TILEXR_UDMA_STATUS_SUCCESS) return 6;
    if (UDMAQuietStatus(&args, 1) != TILEXR_UDMA_STATUS_SUCCESS || std::memcmp(back.data(), src.data(), 512) != 0) return 7;
    // payload, then the signal word
    if (UDMAPutSignalNbiOnQp<unsigned char>(&args, 1, 1, src.data(), 2048, 256, 4088, 77) != TILEXR_UDMA_STATUS_SUCCESS) return 8;
    uint64_t word = 0;
    std::memcpy(&word, region1.data() + 4088, 8);
    if (word != 77 || std::memcmp(region1.data() + 2048, src.data(), 256) != 0) return 9;
    // refused before a byte moves: range, rank, lane, signal alignment, signal range
    std::memset(region1.data(), 0, BYTES);
    if (UDMAPutNbiOnQp<unsigned char>(&args, 1, 0, src.data(), 4000, 512) != TILEXR_UDMA_STATUS_INVALID) return 10;
    if (UDMAPutNbiOnQp<unsigned char>(&args, 0, 0, src.data(), 0, 16) != TILEXR_UDMA_STATUS_INVALID) return 11;
    if (UDMAPutNbiOnQp<unsigned char>(&args, 1, 99, src.data(), 0, 16) != TILEXR_UDMA_STATUS_INVALID) return 12;
    if (UDMAPutSignalNbiOnQp<unsigned char>(&args, 1, 0, src.data(), 0, 16, 4, 1) != TILEXR_UDMA_STATUS_INVALID) return 13;
    if (UDMAPutSignalNbiOnQp<unsigned char>(&args, 1, 0, src.data(), 0, 16, 4096, 1) != TILEXR_UDMA_STATUS_INVALID) return 14;
    if (UDMAGetNbiOnQp<unsigned char>(&args, 1, 0, back.data(), 4090, 16) != TILEXR_UDMA_STATUS_INVALID) return 15;
    for (uint64_t i = 0; i < BYTES; ++i) {
        if (region1[i] != 0) return 16;
    }
    if (SDMAEnabled(&args)) return 17;
    args.extraFlag |= TileXR::TILEXR_FLAG_LOCAL_COPY;
    if (!SDMAEnabled(&args)) return 18;
    std::puts("ok");
    return 0;
}
'''


def test_reference_named_verbs_on_the_host(tmp_path):
    """The reference's device verb names (UDMAPutNbi, UDMAGetNbi, UDMAPutSignalNbi, UDMAQuiet, ...) over the registered-memory
    verbs: round trips between two regions, and every bad rank, lane or range refused before a byte moves.
    (Reference: src/include/tilexr_udma.h:748-1046.)"""
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "udma.cpp"
    src.write_text(UDMA_PROGRAM)
    exe = tmp_path / "udma"
    proc = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc' / 'include'}", str(src), "-o", str(exe)],
                          capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr[-3000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == "ok", (run.returncode, run.stdout, run.stderr)


FEW_ROWS_PROGRAM = r'''
#include <cstdio>
#include "gemm_few_rows.h"
using namespace TileXR;
int main()
{
    const int sms = 148;
    const int64_t sizes[] = {1, 16, 17, 33, 64, 128, 200, 1000};
    const int64_t ns[] = {8, 128, 136, 2048, 7168, 131072}, ks[] = {8, 64, 520, 2048, 4104, 16384};
    const int64_t groupCounts[] = {0, 1, 64, 300}, caps[] = {0, 1, 2, 7, 32, 148, 1000};
    for (int64_t m : sizes) for (int64_t n : ns) for (int64_t k : ks) for (int64_t groups : groupCounts) for (int64_t cap : caps) {
        const int tn = FewRowsTile(m);
        const FewRowsLaunch p = PlanFewRows(m, n, k, groups, tn, sms, cap);
        if (p.grid < 1 || p.grid > 2u * sms || (cap > 0 && p.grid > static_cast<unsigned>(cap))) return 1;      // within the cap
        if (p.split < 1 || p.split > GEMM_SKINNY_MAX_SPLIT || (p.split & (p.split - 1)) != 0 || tn % p.split != 0) return 2;
        if (groups > 0 && p.split != 1) return 3;
        const int64_t kBlocks = (k + 63) / 64, per = (kBlocks + p.split - 1) / p.split;
        if (p.split > 1 && per * (p.split - 1) >= kBlocks) return 4;                                            // no empty part
        if (p.split > 1 && p.grid != ((m + tn - 1) / tn) * ((n + 127) / 128) * p.split) return 5;               // one tile per cluster
    }
    std::puts("ok");
    return 0;
}
'''


def _run_host_program(tmp_path, text, include):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "program.cpp", tmp_path / "program"
    src.write_text(text)
    proc = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{include}", str(src), "-o", str(exe)], capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr[-3000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == "ok", (run.returncode, run.stdout, run.stderr)


def test_few_rows_gemm_keeps_to_the_callers_ctas(tmp_path):
    """The launch of the few-rows GEMM: never more CTAs than a caller allows, and a split of K that leaves no part empty."""
    _run_host_program(tmp_path, FEW_ROWS_PROGRAM, ROOT / "csrc" / "gemm")


FEW_ROWS_LINE_PROGRAM = r'''
#include <cstdio>
#include "gemm_few_rows.h"
int main()
{
    // m, n, k, microseconds of the wide and of the few-rows kernel on a B200
    const struct { int64_t m, n, k; double wide, few; } measured[] = {
        {1, 1024, 4096, 28.2, 9.2},     {16, 8192, 256, 7.1, 7.6},      {16, 16384, 1024, 14.5, 13.5},  {16, 65536, 4096, 94.3, 91.1},
        {24, 1024, 256, 6.7, 8.5},      {32, 16384, 256, 8.3, 10.4},    {24, 256, 512, 8.4, 10.5},      {32, 8192, 512, 9.1, 12.3},
        {17, 7168, 2048, 18.5, 14.0},   {32, 16384, 1024, 14.7, 15.3},  {32, 32768, 4096, 51.7, 51.5},  {64, 4096, 1024, 12.0, 11.8},
        {64, 8192, 2048, 18.6, 16.9},   {64, 16384, 2048, 20.5, 24.6},  {64, 16384, 4096, 35.3, 35.3},  {64, 24576, 4096, 41.3, 45.0},
        {96, 12288, 4096, 35.1, 39.3},  {128, 8192, 2048, 19.9, 23.9},  {128, 8192, 4096, 32.8, 28.9},  {128, 16384, 4096, 37.2, 43.5},
        {128, 32768, 4096, 54.4, 63.9}, {1024, 1024, 4096, 29.0, 25.1}, {256, 4096, 8192, 47.2, 33.6},  {384, 4096, 4096, 29.0, 35.0},
    };
    for (const auto &p : measured) {
        const double taken = TileXR::FewRows(p.m, p.n, p.k) ? p.few : p.wide, other = TileXR::FewRows(p.m, p.n, p.k) ? p.wide : p.few;
        if (taken > other * 1.08) {
            std::printf("%d x %d x %d\n", static_cast<int>(p.m), static_cast<int>(p.n), static_cast<int>(p.k));
            return 1;
        }
    }
    // groups of uneven sizes: rows, groups, microseconds before there was the kernel and with tiles of 16, 32, 64 and 128 rows
    const struct { int64_t rows, groups; double before, t16, t32, t64, t128; } uneven[] = {
        {8, 8, 80.1, 48.4, 49.1, 58.3, 80.5},         {64, 64, 32.0, 15.2, 17.0, 19.3, 20.1},    {512, 64, 37.6, 49.2, 34.1, 29.0, 35.3},
        {1024, 64, 40.8, 69.5, 47.7, 37.4, 35.6},     {512, 8, 45.0, 68.0, 45.8, 39.6, 46.8},    {3072, 64, 35.7, 51.7, 36.5, 35.4, 42.5},
        {16384, 256, 123.2, 282.3, 165.4, 115.6, 101.9},
    };
    for (const auto &p : uneven) {
        const int tn = TileXR::FewRowsGroupTile(p.rows, p.groups);
        const double taken = tn == 16 ? p.t16 : tn == 32 ? p.t32 : tn == 64 ? p.t64 : p.t128;
        if (taken > p.before) {
            std::printf("%d rows, %d groups\n", static_cast<int>(p.rows), static_cast<int>(p.groups));
            return 2;
        }
    }
    std::puts("ok");
    return 0;
}
'''


def test_few_rows_line_lies_where_it_was_measured(tmp_path):
    """The choice between the wide and the few-rows GEMM takes the slower one nowhere by more than the measurements' spread."""
    _run_host_program(tmp_path, FEW_ROWS_LINE_PROGRAM, ROOT / "csrc" / "gemm")


STAGE_COPY_PROGRAM = r'''
#include <cstdio>
#include "gemm_few_rows.h"
int main()
{
    const int64_t counts[] = {0, 1, 1023, 1024, 1025, 100000, 606208, 606209, 10000000};
    for (int64_t vecs : counts) for (int64_t cap : {0, 1, 2, 20, 148, 592, 1000}) {
        const int64_t blocks = TileXR::StageCopyBlocks(vecs, 148, cap);
        if ((blocks == 0) != (vecs == 0) || blocks > 592 || (cap > 0 && blocks > cap) || (blocks - 1) * 1024 >= vecs + (vecs == 0)) return 1;
        if (cap == 0 && blocks < 592 && blocks * 1024 < vecs) return 2;
    }
    std::puts("ok");
    return 0;
}
'''


def test_copy_in_front_of_a_gathered_product_keeps_to_the_callers_ctas(tmp_path):
    _run_host_program(tmp_path, STAGE_COPY_PROGRAM, ROOT / "csrc" / "gemm")


FP8_SLICES_PROGRAM = r'''
#include <cstdio>
#include "gemm_few_rows.h"
int main()
{
    // tiles, blocks of K, microseconds on 74 pairs of a B200 whole and with the last wave in slices of 128, 64 and 32 columns
    const struct { int64_t tiles, blocks; double whole, s128, s64, s32; } measured[] = {
        {2, 4, 7.4, 6.4, 6.0, 5.7}, {2, 64, 32.4, 24.2, 22.9, 22.3}, {8, 16, 12.4, 9.8, 9.3, 9.0}, {16, 4, 7.6, 6.6, 6.0, 8.6},
        {16, 64, 33.0, 24.7, 23.4, 42.0}, {28, 4, 7.8, 6.7, 9.1, 13.7}, {28, 64, 33.9, 25.2, 43.2, 80.1}, {37, 16, 12.8, 10.4, 15.6, 26.5},
        {40, 4, 8.1, 10.0, 11.8, 16.4}, {40, 32, 21.0, 27.3, 35.8, 55.4}, {54, 64, 34.9, 46.7, 63.0, 118.8}, {73, 32, 20.8, 27.9, 46.9, 86.7},
        {76, 4, 12.3, 11.5, 11.2, 11.0}, {76, 64, 64.6, 56.4, 55.0, 54.6}, {90, 16, 22.7, 20.6, 19.7, 25.1}, {114, 32, 37.5, 44.6, 53.2, 72.9},
        {128, 64, 65.2, 77.6, 94.1, 150.1}, {147, 4, 12.9, 15.4, 19.9, 29.3}, {150, 32, 53.8, 49.4, 48.4, 48.2}, {188, 64, 99.7, 109.7, 126.1, 162.6},
        {224, 4, 21.9, 20.9, 20.6, 20.5}, {224, 32, 70.2, 66.0, 65.1, 64.9}, {276, 64, 137.4, 146.6, 160.0, 214.7}, {448, 16, 70.4, 68.2, 67.7, 67.9},
        {448, 64, 230.3, 226.5, 223.7, 225.2},
    };
    for (const auto &p : measured) {
        const int width = TileXR::PlanFp8Slices(p.tiles, 74).width;
        const double taken = width == 32 ? p.s32 : width == 64 ? p.s64 : width == 128 ? p.s128 : p.whole;
        for (double other : {p.whole, p.s128, p.s64, p.s32}) {
            if (taken > other * 1.02) {
                std::printf("%d tiles, %d blocks of K\n", static_cast<int>(p.tiles), static_cast<int>(p.blocks));
                return 1;
            }
        }
    }
    for (int64_t pairs : {1, 2, 7, 74, 148}) for (int64_t tiles = 1; tiles <= 500; ++tiles) {
        const TileXR::Fp8Slices s = TileXR::PlanFp8Slices(tiles, pairs);
        if (s.wide < 0 || s.wide > tiles || (s.items - s.wide) * s.width != (tiles - s.wide) * 256) return 2;     // every column of every tile once
        if ((s.items + pairs - 1) / pairs != (tiles + pairs - 1) / pairs) return 3;                                // no wave more than whole tiles take
    }
    std::puts("ok");
    return 0;
}
'''


def test_slices_of_the_block_scaled_product_lie_where_they_were_measured(tmp_path):
    """The choice is the fastest one of every row, within 2 %, the spread of the measurements."""
    _run_host_program(tmp_path, FP8_SLICES_PROGRAM, ROOT / "csrc" / "gemm")

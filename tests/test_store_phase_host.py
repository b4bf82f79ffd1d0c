"""The store phase of a paired tile (fold_and_store), compiled for the host with the device's primitives stood in: a warp is 32
threads. Every variable starts out filled with a pattern, so a value that is read before it is written, or after the variable it
was written to has gone, shows in the result."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bsipytorch_b200", "csrc")

HARNESS = r"""
#include <barrier>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
struct alignas(16) uint4 { uint32_t x, y, z, w; };
static uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
struct Map { int bytes; };
using CUtensorMap = Map;
struct Finishing { int relu, scaled_cols; float factor; const void* add; int64_t ld_add; };
static thread_local struct { unsigned x; } threadIdx;
static std::barrier<> warp(32);
static void __syncwarp() { warp.arrive_and_wait(); }
static bool elect_one() { return threadIdx.x == 0; }
static uint64_t pack2(float, float) { return 0; }
static int __float2int_rn(float v) { return static_cast<int>(v); }
static int __float_as_int(float v) { int i; memcpy(&i, &v, 4); return i; }
static float __fmaf_rn(float a, float b, float c) { return a * b + c; }
static float int_to_float_exact(int v) { return static_cast<float>(v); }
static int accumulator(int row, int col) { return row * 7 + col * 3 - 500; }
static void tmem_ld32(uint32_t t, int32_t (&r)[32]) { for (int e = 0; e < 32; ++e) r[e] = accumulator(threadIdx.x, t + e); }
static void tmem_ld16(uint32_t t, int32_t (&r)[32]) { for (int e = 0; e < 16; ++e) r[e] = accumulator(threadIdx.x, t + e); }
static void tmem_ld_wait_for(int32_t (&)[32]) {}
static void tc_fence_before() {}
template <typename T> T behind_wait(T p) { return p; }
alignas(16) static uint8_t shared_memory[8 * 4096];
static uint32_t smem_u32(const void* p) { return static_cast<const uint8_t*>(p) - shared_memory; }
// a piece of 16 bytes: integers, so that a sum needs no rounding
template <typename OutT> uint4 finish16(const float* f, const float*, const OutT*, uint64_t, bool, bool) {
    OutT o[16 / sizeof(OutT)];
    for (size_t i = 0; i < 16 / sizeof(OutT); ++i) o[i] = static_cast<OutT>(static_cast<int>(f[i]));
    uint4 r;
    memcpy(&r, o, 16);
    return r;
}
static uint4 finish16_plain(const float* f, const float* w, uint64_t s) { return finish16<int32_t>(f, w, nullptr, s, false, false); }
template <typename OutT> uint4 plus16(uint4 a, uint4 b, OutT) {
    OutT x[16 / sizeof(OutT)], y[16 / sizeof(OutT)];
    memcpy(x, &a, 16);
    memcpy(y, &b, 16);
    for (size_t i = 0; i < 16 / sizeof(OutT); ++i) x[i] += y[i];
    memcpy(&a, x, 16);
    return a;
}
template <typename OutT> uint4 times(uint4 a, float, OutT) { return a; }
static std::vector<uint8_t> output;
static int out_rows, out_cols, out_size;
static void tma_store_2d(const CUtensorMap* map, uint32_t at, int col, int row) {      // rows of 128 or 64 bytes, swizzled
    for (int r = 0; r < 32 && row + r < out_rows; ++r)
        for (int c = 0; c < map->bytes / out_size && col + c < out_cols; ++c) {
            const int ch = c * out_size / 16, to = map->bytes == 128 ? ch ^ (r & 7) : ch ^ ((r >> 1) & 3);
            memcpy(&output[(static_cast<size_t>(row + r) * out_cols + col + c) * out_size],
                   shared_memory + at + r * map->bytes + to * 16 + c * out_size % 16, out_size);
        }
}
@SOURCE@
template <typename OutT, int kCols, bool ADD>
int wrong(int Q, int R, int col, int kind) {
    out_rows = Q; out_cols = R; out_size = sizeof(OutT);
    output.assign(static_cast<size_t>(Q) * R * sizeof(OutT), 0xcc);
    std::vector<OutT> add(static_cast<size_t>(Q) * R);
    for (size_t i = 0; i < add.size(); ++i) add[i] = static_cast<OutT>(i * 2654435761u >> 9);
    const Map whole{128}, tail{64};
    const Finishing fin{0, 0, 1.0f, ADD ? add.data() : nullptr, R};
    std::vector<std::thread> lanes;
    for (unsigned lane = 0; lane < 32; ++lane)
        lanes.emplace_back([&, lane] {
            threadIdx.x = lane;
            float acc[kCols];
            for (int e = 0; e < kCols; ++e) {
                const int sum = 1000 - e;
                if (kind == kFloatSums) acc[e] = static_cast<float>(sum);
                else memcpy(&acc[e], &sum, 4);
            }
            float w[kCols] = {};
            OutT b[kCols] = {};
            fold_and_store<OutT, kCols, ADD>(acc, 0u, 2.0f, kind, shared_memory, w, b, whole, tail, 0, Q, col, R, 1.0f, true, false, fin, [] {});
        });
    for (std::thread& t : lanes) t.join();
    int bad = 0;
    for (int r = 0; r < Q && r < 32; ++r)
        for (int c = col; c < R && c < col + kCols; ++c) {
            OutT got;
            memcpy(&got, &output[(static_cast<size_t>(r) * R + c) * sizeof(OutT)], sizeof(OutT));
            const OutT sum = static_cast<OutT>(accumulator(r, c - col) * 2 + 1000 - (c - col));
            bad += got != static_cast<OutT>(sum + (ADD ? add[static_cast<size_t>(r) * R + c] : OutT(0)));
        }
    return bad;
}
template <typename OutT, bool ADD>
void widths(const char* name) {
    for (int kind = 0; kind < 3; ++kind)
        for (int narrow = 0; narrow < 2; ++narrow) {      // a whole tile; one clipped in both directions
            const int Q = narrow ? 19 : 32, less = narrow ? 8 : 0;
            printf("%s %d %d: %d %d %d\n", name, kind, narrow, wrong<OutT, 32, ADD>(Q, 64 + 32 - less, 64, kind),
                   wrong<OutT, 64, ADD>(Q, 64 + 64 - less, 64, kind), wrong<OutT, 128, ADD>(Q, 64 + 128 - less, 64, kind));
        }
}
int main() {
    widths<int16_t, true>("16 bits with a sum");
    widths<int16_t, false>("16 bits");
    widths<int32_t, true>("32 bits with a sum");
    widths<int32_t, false>("32 bits");
}
"""


def test_store_phase_reads_what_it_has_written(tmp_path):
    text = open(os.path.join(CSRC, "dot_tcgen05_pair.cuh")).read()
    found = re.search(r"^enum SumKind.*?^}\n", text, re.S | re.M)
    assert found and "void fold_and_store" in found.group(0)
    source = re.sub(r"asm volatile\(.*?\);", "", found.group(0))
    (tmp_path / "store.cpp").write_text(HARNESS.replace("@SOURCE@", source))
    subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-fno-strict-aliasing", "-ftrivial-auto-var-init=pattern", "-o", str(tmp_path / "store"),
                    str(tmp_path / "store.cpp")], check=True)
    lines = subprocess.run([str(tmp_path / "store")], check=True, capture_output=True, text=True, timeout=120).stdout.splitlines()
    assert len(lines) == 24
    assert [l for l in lines if not l.endswith(": 0 0 0")] == []

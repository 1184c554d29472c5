"""The prefill GEMM's pipeline on the CPU: its roles' own code, compiled for the host with barriers that record,
gives the order in which each role waits and hands over; those orders are then played against one another on
mbarriers (a wait knows a phase by its parity only) with each role in turn as late as it can be."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tianchen-rv_b200", "csrc")

COMMON = r"""
#pragma once
#include <cstddef>
#include <cstdint>
#include <cstdio>
#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __grid_constant__
#define __shared__
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) ulonglong2 { uint64_t x, y; };
struct Index { unsigned x; };
static Index threadIdx, blockIdx, gridDim;
struct CUtensorMap {};
namespace tcrv {
constexpr int kQK = 32, kDevErrBarrierTimeout = 1;
struct DeviceErrorWords {};
inline void raise_device_error(const DeviceErrorWords &, int) {}
inline void say(const char *what, const uint64_t *bar, uint32_t parity) { std::printf("%s %d %u\n", what, static_cast<int>(reinterpret_cast<uintptr_t>(bar) / 8), parity); }
inline uint32_t smem_addr(const void *) { return 0; }
inline void mbar_init(uint64_t *, uint32_t) {}
inline void mbar_fence_init() {}
inline void mbar_arrive(uint64_t *bar) { say("arrive", bar, 0); }
inline void mbar_arrive_if(uint64_t *bar, bool pred) { if (pred) mbar_arrive(bar); }
inline void mbar_arrive_expect_tx(uint64_t *, uint32_t) {}
inline bool mbar_test(uint64_t *, uint32_t) { return false; }
inline bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, volatile uint32_t * = nullptr) { say("wait", bar, parity); return true; }
inline void umma_commit(uint64_t *bar) { say("arrive", bar, 0); }
inline void tma_load_2d(void *, const CUtensorMap *, int, int, uint64_t *) {}
inline void prefetch_tensormap(const CUtensorMap *) {}
inline void tmem_alloc(uint32_t *, uint32_t) {}
inline void tmem_relinquish_alloc_permit() {}
inline void tmem_dealloc(uint32_t, uint32_t) {}
inline void tcgen05_fence_before_thread_sync() {}
inline void tcgen05_fence_after_thread_sync() {}
inline uint64_t umma_desc_k_major_sw128(uint32_t) { return 0; }
inline bool elect_one() { return true; }
constexpr uint32_t umma_idesc_e4m3(int, int) { return 0; }
template <typename... A> inline void umma_f8_first(A...) { std::printf("fill\n"); }
template <typename... A> inline void umma_f8_again(A...) { std::printf("use\n"); }
template <int N> inline void tmem_ld_32x32b(uint32_t, uint32_t *v) { for (int i = 0; i < N; ++i) v[i] = 0; }
inline void tmem_ld_wait() {}
}  // namespace tcrv
inline void __syncwarp() {}
inline void __syncthreads() {}
inline bool __all_sync(uint32_t, bool v) { return v; }
template <typename T> inline T __shfl_sync(uint32_t, T v, int) { return v; }
inline float __uint_as_float(uint32_t) { return 0.0f; }
// the header's inline PTX: none of it is part of the pipeline
#define asm(...) ((void)0)
#define volatile(...) ("")
"""

# argv: multi (0, 1), columns of a narrow item (0: none), blocks per row, then the items: w(hole) or h(alf)
MAIN = r"""
#include "gemm_tc.cuh"
#include <cstdlib>
#include <vector>
using namespace tcrv;
template <bool kMulti, int kNarrow>
void roles(uint32_t nb, int count, char **items) {
  using Plan = GemmPlan<kNarrow>;
  constexpr int kStages = GemmSmem<kMulti, kNarrow>::kStages;
  std::printf("stages %d %d\n", kStages, Plan::kTmemStages);
  std::vector<uint8_t> stages(GemmSmem<kMulti, kNarrow>::kBytes + 16);
  GemmArgs a = {};
  a.nb = nb;
  for (int role = -1; role < kGemmMmaWarps; ++role) {
    std::printf("role %d\n", role);
    GemmEpilogueCtx c = {};
    c.stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(stages.data()) + 15) / 16 * 16);
    c.smem_full = reinterpret_cast<uint64_t *>(8 * 0);  // recorded, never read
    c.smem_empty = reinterpret_cast<uint64_t *>(8 * 100);
    c.tmem_full = reinterpret_cast<uint64_t *>(8 * 200);
    c.tmem_empty = reinterpret_cast<uint64_t *>(8 * 300);
    c.mma_warp = role;
    for (int i = 0; i < count; ++i) {
      const GemmItem it = {0, 0, items[i][0] == 'w'};
      if (role < 0 && it.whole)
        gemm_epilogue_item<Plan, typename Plan::Full, false, false, kStages>(a, c, it, 0, 0);
      else if (role < 0)
        gemm_epilogue_item<Plan, typename Plan::Half, false, false, kStages>(a, c, it, 0, 0);
      else if (it.whole)
        gemm_mma_item<Plan, typename Plan::Full, kStages>(a, c, 0, true);
      else
        gemm_mma_item<Plan, typename Plan::Half, kStages>(a, c, 0, true);
    }
  }
}
int main(int argc, char **argv) {
  const uint32_t nb = std::atoi(argv[3]);
  const int narrow = std::atoi(argv[2]);
  if (argv[1][0] == '1')
    roles<true, 0>(nb, argc - 4, argv + 4);
  else if (narrow == 0)
    roles<false, 0>(nb, argc - 4, argv + 4);
  else if (narrow == 16)
    roles<false, 16>(nb, argc - 4, argv + 4);
  else
    roles<false, 32>(nb, argc - 4, argv + 4);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("gemm_pipeline")
    shutil.copy(os.path.join(CSRC, "gemm_tc.cuh"), d)
    (d / "tcrv_common.cuh").write_text(COMMON)
    (d / "tcgen05.cuh").write_text('#include "tcrv_common.cuh"\n')
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-w", "-std=c++17", "-o", d / "roles", d / "main.cpp"], check=True)
    return d / "roles"


def record(program, multi, narrow, nb, items):
    """(shared-memory stages, TMEM stages, {role: [(what, barrier, parity)]}) of the epilogue (-1) and the MMA warps (0, 1)."""
    out = subprocess.run([program, str(multi), str(narrow), str(nb), *items], check=True, capture_output=True, text=True).stdout
    stages, tmem, roles = 0, 0, {}
    for line in out.splitlines():
        what, number, parity = (line.split() + ["0", "0"])[:3]
        if what == "stages":
            stages, tmem = int(number), int(parity)
        elif what == "role":
            trace = roles.setdefault(int(number), [])
        else:
            trace.append((what, int(number), int(parity)))
    return stages, tmem, roles


def play(roles, late):
    """Every role runs as far as it can before `late` makes one step; the roles that never finish."""
    arrived, at = {}, dict.fromkeys(roles, 0)  # arrivals at a barrier; next step of a role
    filled = [None]  # whose A operand is in the tensor core's buffer

    def step(role):
        if at[role] == len(roles[role]):
            return False
        what, bar, parity = roles[role][at[role]]
        if what == "arrive":
            arrived[bar] = arrived.get(bar, 0) + 1
        elif what == "fill":
            filled[0] = role
        elif what == "use":
            assert filled[0] == role, "another warp's MMA came between the two that share an operand"
        elif arrived.get(bar, 0) // (2 if bar // 100 == 3 else 1) % 2 == parity:  # free accumulators: epilogue and turn
            return False
        at[role] += 1
        return True

    while any([step(r) for r in roles if r != late]) or step(late):
        pass
    return [r for r in roles if at[r] < len(roles[r])]


@pytest.mark.parametrize("multi,narrow,nb,items", [
    (0, 0, 40, "ww"), (0, 0, 40, "hh"), (0, 0, 41, "whwh"), (0, 0, 1, "whhwhhh"), (1, 0, 40, "whh"), (0, 32, 40, "www"), (0, 16, 61, "www"),
    (0, 32, 1, "wwwwwwwwwwwwwwwwwwwwww"),
])
def test_no_role_can_come_too_late_for_a_phase(program, multi, narrow, nb, items):
    stages, tmem, roles = record(program, multi, narrow, nb, items)
    fills = (nb + 3) // 4 * len(items)
    # one epilogue warp stands for the eight, which do the same; the producer fills stage after stage; before the
    # first item the epilogue hands over all accumulators and the first MMA warp gives itself the first turn
    roles[-1][:0] = [("arrive", 300 + i, 0) for i in range(tmem)]
    roles[0][:0] = [("arrive", 300, 0)]
    roles["producer"] = [e for i in range(fills) for e in (("wait", 100 + i % stages, 1 - i // stages % 2), ("arrive", i % stages, 0))]
    for late in roles:
        assert play(roles, late) == [], f"role {late} comes too late"

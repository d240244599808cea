// gb_inv_warp.cuh with a warp's lanes as contexts that take turns, for test_inv_warp.py: values
// to invert (hex words, one a line) on standard input, "<field> <value>", their
// inverses by the division steps alone on standard output; every lane's result
// has to be the same.
#include <stdio.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <functional>
#include <vector>

#include "gb_field.cuh"

#define GB_WARP_ON_HOST
#define __device__
#define __constant__
#define __forceinline__ inline
#define __noinline__

static struct { unsigned x; } threadIdx;
static ucontext_t lane_context[32], caller;
static int64_t warp_value[32];
static std::function<void()> lane_work;

// on to the next lane, and back here when the others have had their turn
static void turn()
{
    const unsigned me = threadIdx.x, next = (me + 1) % 32;
    swapcontext(&lane_context[me], &lane_context[next]);
    threadIdx.x = me;
}

static void lane_main(int lane)
{
    threadIdx.x = (unsigned)lane;
    lane_work();
    // lanes end in order, as they take part in the same exchanges
    if (lane < 31) setcontext(&lane_context[lane + 1]);
    setcontext(&caller);
}

static void run_warp(std::function<void()> work)
{
    static std::vector<char> stacks(32 << 18);
    lane_work = work;
    for (int lane = 0; lane < 32; lane++) {
        getcontext(&lane_context[lane]);
        lane_context[lane].uc_stack.ss_sp = stacks.data() + ((size_t)lane << 18);
        lane_context[lane].uc_stack.ss_size = 1 << 18;
        lane_context[lane].uc_link = nullptr;
        makecontext(&lane_context[lane], (void (*)())lane_main, 1, lane);
    }
    swapcontext(&caller, &lane_context[0]);
}

template <class T>
static T warp_exchange(T v, unsigned from)
{
    warp_value[threadIdx.x] = (int64_t)v;
    turn();
    const T r = from < 32 ? (T)warp_value[from] : v;
    turn();
    return r;
}
template <class T>
static T __shfl_sync(unsigned, T v, int lane) { return warp_exchange(v, (unsigned)lane); }
template <class T>
static T __shfl_up_sync(unsigned, T v, unsigned off) { return warp_exchange(v, threadIdx.x - off); }
template <class T>
static T __shfl_down_sync(unsigned, T v, unsigned off) { return warp_exchange(v, threadIdx.x + off); }
static unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s)
{
    return (unsigned)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
using std::min;
static int __ffs(int v) { return __builtin_ffs(v); }

#include "gb_inv_warp.cuh"

template <class Cfg>
static bool invert(const char *hex)
{
    gb::mont_t<Cfg> a;
    for (int i = 0; i < Cfg::N; i++) {
        char word[9] = {0};
        memcpy(word, hex + 8 * (Cfg::N - 1 - i), 8);
        unsigned v;
        if (sscanf(word, "%8x", &v) != 1) return false;
        a.v[i] = v;
    }
    gb::mont_t<Cfg> out[32];
    run_warp([&] { out[threadIdx.x] = gb::inverse_steps<Cfg>(&a); });
    for (int lane = 1; lane < 32; lane++)
        if (memcmp(&out[lane], &out[0], sizeof(out[0]))) return false;
    for (int i = Cfg::N - 1; i >= 0; i--) printf("%08x", out[0].v[i]);
    printf("\n");
    return true;
}

int main()
{
    char field[3], hex[128];
    while (scanf("%2s %127s", field, hex) == 2)
        if (!(field[1] == 'p' ? invert<gb::FpCfg>(hex) : invert<gb::FrCfg>(hex))) return 1;
    return 0;
}

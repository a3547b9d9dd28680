// Shared by the reductions that keep a matrix's rows on the CTAs of one
// cooperative launch (bidiag.cu, hess.cu): warp sums, and the tagged slots in
// which values cross the CTAs.
#pragma once
#include "jlc_device.cuh"

namespace jlc {

__device__ __forceinline__ double shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += shfl_xor(v, o);
    return v;
}

// Eight per-lane values summed over the warp: on return lane 4 i holds the
// sum of value i (a halving exchange, then two butterfly steps).
__device__ __forceinline__ double warp_sum8(double (&v)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double keep = (lane & 16) ? v[i + 4] : v[i], give = (lane & 16) ? v[i] : v[i + 4];
        v[i] = keep + shfl_xor(give, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double keep = (lane & 8) ? v[i + 2] : v[i], give = (lane & 8) ? v[i] : v[i + 2];
        v[i] = keep + shfl_xor(give, 8);
    }
    const double keep = (lane & 4) ? v[1] : v[0], give = (lane & 4) ? v[0] : v[1];
    double s = keep + shfl_xor(give, 4);
    s += shfl_xor(s, 2);
    s += shfl_xor(s, 1);
    return s;
}

// Values exchanged between CTAs of one cooperative launch without a barrier:
// a slot is 16 bytes, the value and a word that carries the tag of its use
// and a small integer.  It is written and read by single 128-bit accesses at
// gpu scope, so a reader that finds the tag has the value: the data is its
// own flag, and an exchange costs one store and one load through L2 instead of
// store, fence, counter, poll and load.  Tags grow from use to use; slots are
// zeroed before the launch and tag 0 is never waited for.
struct __align__(16) Slot {
    double v;
    unsigned lo, tag;
};

__device__ __forceinline__ void slot_put(Slot* s, double v, unsigned tag, int aux) {
    const unsigned long long hi = ((unsigned long long)tag << 32) | (unsigned)aux;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(s),
                 "l"(__double_as_longlong(v)), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ void slot_load(const Slot* s, double& v, unsigned& tag, int& aux) {
    long long lo;
    unsigned long long hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(s)
                 : "memory");
    v = __longlong_as_double(lo);
    tag = (unsigned)(hi >> 32);
    aux = (int)(unsigned)hi;
}

// the value of a slot this thread has already waited for
__device__ __forceinline__ double slot_value(const Slot* s) {
    double v;
    unsigned tag;
    int aux;
    slot_load(s, v, tag, aux);
    return v;
}

// A wait's occasional check, out of line so that the waits stay small: given
// the time the wait began (0 at the first check), returns it, or 0 once the
// limit has passed (which it records) or an error is recorded.
static __device__ __noinline__ uint64_t slot_check(uint64_t t0, int* status) {
    const uint64_t now = globaltimer_ns();
    if (*(volatile int*)status != 0) return 0;
    if (t0 == 0) return now;
    if (now - t0 <= wait_limit_ns(status)) return t0;
    atomicOr(status, JLC_DEV_TIMEOUT);
    return 0;
}

// Waits until every one of the N slots carries `tag` and takes their values
// (and integers): all loads of a round are in flight together.  Bounded like
// mbar_wait: false once the wait limit has passed or an error is recorded.
template <int N>
__device__ __forceinline__ bool slot_wait(const Slot* const (&s)[N], unsigned tag, double (&v)[N], int* status,
                                          int* aux = nullptr) {
    uint64_t t0 = 0;
    unsigned it = 0;
#pragma unroll 1
    for (;;) {
        unsigned bad = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            unsigned tg;
            int ax;
            slot_load(s[i], v[i], tg, ax);
            if (aux) aux[i] = ax;
            bad |= tg ^ tag;
        }
        if (bad == 0) return true;
        if ((++it & 255u) == 0u && (t0 = slot_check(t0, status)) == 0) return false;
    }
}

// The slots of columns j0 + tid + i BT < n of this thread (past the last column
// the values mean nothing).  A warp without a column does not poll, and for a
// block past the last column it polls its first one again: were they to poll
// the last column's slot, every warp of every CTA would, and its L2 slice
// serves those requests one by one (bidiagonalisation 1152 x 1024: 6.8 us a
// step against 5.3).
template <int BT, int N>
__device__ __forceinline__ bool slot_wait_columns(const Slot* s, int j0, int n, unsigned tag, double (&v)[N],
                                                  int* status) {
    const int first = j0 + (int)(threadIdx.x & ~31u);  // of this warp
    if (first >= n) return true;
    const Slot* at[N];
#pragma unroll
    for (int i = 0; i < N; ++i) at[i] = s + min(j0 + (int)threadIdx.x + (first + i * BT < n ? i * BT : 0), n - 1);
    return slot_wait(at, tag, v, status);
}

}  // namespace jlc

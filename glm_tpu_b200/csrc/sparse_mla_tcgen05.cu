// Sparse absorbed-MLA attention of many query rows (prefill) on the 5th-generation tensor cores: 64 heads, latent 512, rotary 64.
//
// A query row attends to its own list of up to top_k cache rows, so the only operand that is shared is the row's 64 heads.  The KEYS are
// therefore the M of both products (128 gathered keys, then 128 latent columns) and the heads the N:
//
//   S^T [128 keys x 64 heads]    = K Q^T     A = gathered rows, K-major;     B = the row's queries, K-major
//   O^T [4 x 128 columns x 64]  += V^T P^T   A = the same gathered rows, MN-major;  B = weights [key][head], MN-major
//
// so that a full 128-row instruction is filled although a row has 64 heads, one gather of 1,152 bytes a key feeds both products of all
// heads, and a thread of the softmax owns a key (a TMEM lane) with the scores of half the heads.
//
//   warps 0-7   softmax: scores from TMEM (two threads per key, 32 heads each), weights to shared memory, output of a finished row
//   warps 8-11  gather: cp.async of the selected rows into nine 128-key x 64-column boxes (128-byte swizzle); queries by TMA.  Then, while the
//               weights are made, the output so far is scaled to the new maxima
//   warp 12     issues every tcgen05.mma, owns the TMEM
//
// What bounds it: the gather (147 KB per 128 keys and row out of L2) and the chain gather -> S -> softmax -> O of a block, because the
// queries (72 KB) leave room for one block of keys.  The chain is shortened by freeing the boxes two by two and handing them on two by two: the next
// block's first columns are on their way, and multiplied with the queries, while the last columns of this block are still in use.  The weights lie where
// the rotary columns were, which the second product does not need.  Of 10.6 k clocks a block (128 keys) the gather waited 7.2 k for boxes to be freed
// and the softmax worked 3.0 k, a quarter of that on the output's scale, which changes in nine blocks of ten; a row's division and stores took 14.5 k.
// 2,048 rows of 2,048 keys: 1,276 us; pairs handed on as they arrive, not behind the last copy that is asked for, 1,126 (two pairs later 1,173; eight
// gather warps, which leave the softmax 96 registers, 1,181); with the scaling in the gather warps and divisions without branches 1,009.
//
// Weights are taken relative to the running maximum of their head, block by block, as in sparse_mla_rows_kernel (which takes every other
// shape): the heaviest weight is then 1 and loses nothing when the weights enter the second product as bf16.  A reference that lags behind by up
// to 2^8 saves the reduction, but rounds the heaviest weight too: against 64 bits, 2,048 keys, queries of standard deviation 4, the result is
// then 2.12e-3 off, here and by sparse_mla_rows_kernel 1.73e-3.  Sums of weights stay per thread until the row ends.  Scores, exponents and
// sums are fp32.
//
// Rows are dealt to one CTA per SM, longest (last) first.  2,048 rows of 2,048 keys on a B200: 5.27 ms with sparse_mla_rows_kernel (111 TFLOP/s),
// 1.01 ms here (579 TFLOP/s); 777 rows 0.44 ms; 64 rows 79 us; 200 rows of 200 keys: 84 -> 26.
//
// Every wait is bounded; a wait that runs out raises GLMB_STATUS_WAIT_TIMEOUT and the CTA still releases its TMEM.
#include "attention_core.cuh"
#include "tcgen05.cuh"

#define SM_H 64
#define SM_HALF 32     // heads of a softmax thread
#define SM_L 512
#define SM_W 576
#define SM_KEYS 128
#define SM_BOXES 9
#define SM_KBOX 16384  // bytes of 128 keys x 64 columns
#define SM_QBOX 8192   // bytes of 64 heads x 64 columns
#define SM_THREADS 416
#define SM_SMEM (SM_BOXES * (SM_KBOX + SM_QBOX) + 1024)
#define SM_LOG2E 1.4426950408889634f

__device__ __forceinline__ void sm_ld32(uint32_t taddr, float* r) {
    uint32_t v[32];
    tmem_ld32(taddr, v);
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __uint_as_float(v[i]);
}
__device__ __forceinline__ void sm_st32(uint32_t taddr, const float* r) {
#define V(i) "r"(__float_as_uint(r[i]))
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), V(0), V(1), V(2), V(3), V(4), V(5), V(6), V(7), V(8), V(9), V(10), V(11), V(12), V(13), V(14), V(15), V(16), V(17), V(18),
        V(19), V(20), V(21), V(22), V(23), V(24), V(25), V(26), V(27), V(28), V(29), V(30), V(31) : "memory");
#undef V
}
// MN-major operand, 128-byte swizzle: 64 columns (128 bytes) per K row, 8 K rows per 1024-byte group, 64-column boxes SM_KBOX apart.
__device__ __forceinline__ uint64_t sm_desc_mn(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(SM_KBOX >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ float sm_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// a / b, rounded correctly for |a| of 2^-100 and more and b from 1 to 2^100 (the contract divides), of y = the rounded 1 / b: a quotient and one correction by its
// remainder (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990), without the branch of a division (2,048 rows of 2,048 keys
// 1,060 us with it).  The rounding of y moves a * y by less than an ulp: the first quotient is within 1.5 ulp of a / b, and next to a midpoint of two
// numbers it is one of the two.  There its remainder, of half an ulp, is exact, and y's error moves the corrected sum by less than 2^-25 ulp, while a / b, which cannot
// be a midpoint, is 2^-24 ulp / (b / 2^exponent) from it at least.  240 million quotients next to midpoints gave no other result than the division.
// Infinities keep the first quotient.
__device__ __forceinline__ float sm_quotient(float a, float b, float y) {
    const float q = a * y, exact = fmaf(fmaf(-q, b, a), y, q);
    return exact == exact ? exact : q;
}
__device__ __forceinline__ void sm_barrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
struct SparseMlaArgs {
    const bf16* kv_cache;
    const int* sel_local;   // [rows, top_k]
    const int* sel_counts;  // [rows, 2]: the second is the number of entries
    const int* row_lane;
    bf16* o_lat;            // [rows, 64, 512]
    int rows, layer, layers, local_cap, top_k;
    float scale;
    uint32_t* status;
};

__global__ void __launch_bounds__(SM_THREADS, 1) sparse_mla_tc_kernel(const __grid_constant__ CUtensorMap map_q, SparseMlaArgs a) {
    GLMB_PDL_PROLOGUE();  // before the TMEM allocation: a kernel still running may need the columns to finish
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(16) float top_s[8][SM_HALF], ref_s[8][SM_HALF], fix_s[8][SM_HALF], sum_s[8][SM_HALF], inv_s[8][SM_HALF];  // per softmax warp and head of its half
    __shared__ __align__(8) uint64_t q_full, k_full[5], s_full, fix_full, p_full, o_done[4];
    __shared__ uint32_t tmem_slot;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    unsigned char* k_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = k_s + SM_BOXES * SM_KBOX;
    unsigned char* p_s = k_s + (SM_BOXES - 1) * SM_KBOX;  // the rotary box

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1); mbar_init(&s_full, 1); mbar_init(&fix_full, 2); mbar_init(&p_full, 12);
        for (int i = 0; i < 5; ++i) mbar_init(k_full + i, 4);
        for (int i = 0; i < 4; ++i) mbar_init(o_done + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;  // S^T at columns 0..63, O^T of column block j at 64 + 64 j
    auto keys_of = [&](int r) { return min(max(a.sel_counts[2 * r + 1], 0), a.top_k); };

    uint32_t n = 0;  // blocks of keys so far, over the rows of this CTA: the phase of every barrier but q_full
    if (warp >= 8 && warp < 12) {
        // ---- gather: thread (key % 16, piece) copies 16 bytes of eight keys per box ---------------------------------------
        const int tid = threadIdx.x - 256, piece = tid & 7, key0 = tid >> 3;
        unsigned char* dst0 = k_s + (key0 >> 3) * 1024 + (key0 & 7) * 128 + ((piece ^ (key0 & 7)) << 4);
        // the places of the next block's keys are asked for a block ahead: a load that the copies wait for would cost every block its latency
        int next[8], next_i = blockIdx.x, next_start = 0;
        auto fetch = [&]() {
            while (next_i < a.rows && next_start >= keys_of(a.rows - 1 - next_i)) { next_i += gridDim.x; next_start = 0; }
            if (next_i >= a.rows) return;
            const int r = a.rows - 1 - next_i, cnt = keys_of(r) - next_start;
            const int* list = a.sel_local + (int64_t)r * a.top_k + next_start + key0;
#pragma unroll
            for (int e = 0; e < 8; ++e) next[e] = key0 + 16 * e < cnt ? list[16 * e] : 0;
            next_start += SM_KEYS;
        };
        fetch();
        auto hand_on = [&](int j) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies -> visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(k_full + j);
        };
        bool ok = true;
        for (int i = blockIdx.x; i < a.rows && ok; i += gridDim.x) {
            const int r = a.rows - 1 - i, count = keys_of(r);
            const bf16* cache = a.kv_cache + ((int64_t)a.row_lane[r] * a.layers + a.layer) * (int64_t)a.local_cap * SM_W + piece * 8;
            for (int start = 0; start < count && ok; start += SM_KEYS, ++n) {
                const int cnt = min(SM_KEYS, count - start), used = (cnt + 15) & ~15;  // the second product reads keys in sixteens
                const bf16* src[8];
                bool bad = false;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    bad |= (unsigned)next[e] >= (unsigned)a.local_cap;
                    src[e] = cache + (int64_t)min(max(next[e], 0), a.local_cap - 1) * SM_W;
                }
                if (bad) raise_status(a.status, GLMB_STATUS_BAD_INDEX);
                fetch();
                for (int j = 0; j < 5; ++j) {  // box pairs 0-1, 2-3, 4-5, 6-7, then the rotary box, which holds the weights until the end
                    if (n > 0 && !mbar_wait_warp(o_done + min(j, 3), (n - 1) & 1)) { ok = false; break; }
                    if (j == 0 && start == 0 && tid == 0) {  // the products of the row before are done with its queries
                        mbar_expect_tx(&q_full, SM_BOXES * SM_QBOX);
                        for (int b = 0; b < SM_BOXES; ++b) tma_load_2d(q_s + b * SM_QBOX, &map_q, &q_full, b * 64, r * SM_H);
                    }
                    for (int b = 2 * j; b < min(2 * j + 2, SM_BOXES); ++b)
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (key0 + 16 * e < used) {
                                const uint32_t dst = smem_u32(dst0 + b * SM_KBOX + e * 2048);
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src[e] + b * 64), "r"(key0 + 16 * e < cnt ? 16 : 0) : "memory");
                            }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    if (j > 0) {  // a pair is handed on when the next one has been asked for: the products with it run while later boxes are still in use
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                        hand_on(j - 1);
                    }
                }
                if (!ok) break;
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                hand_on(4);
                // ---- the output so far to the new maxima of its heads, while the softmax warps make the weights: nothing is to be copied meanwhile
                if (start > 0) {
                    if (!mbar_wait_warp(&fix_full, n & 1)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                    for (int half = 0; half < 2; ++half) {
                        const float* fix = fix_s[half * 4];
                        if (!__any_sync(0xffffffffu, fix[lane] != 1.f)) continue;
                        const uint32_t o_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 64 + half * SM_HALF;
#pragma unroll 1
                        for (int c = 0; c < SM_L / 2; c += 64) {
                            float o[SM_HALF];
                            sm_ld32(o_addr + c, o);
#pragma unroll
                            for (int e = 0; e < SM_HALF; ++e) o[e] *= fix[e];
                            sm_st32(o_addr + c, o);
                        }
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(&p_full);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 12) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(SM_KEYS, SM_H), idesc_o = umma_idesc_bf16(128, SM_H) | (1u << 15) | (1u << 16);  // both MN-major
        const uint32_t k_addr = smem_u32(k_s), q_addr = smem_u32(q_s), p_addr = smem_u32(p_s);
        uint32_t row_n = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < a.rows && ok; i += gridDim.x) {
            const int count = keys_of(a.rows - 1 - i);
            for (int start = 0; start < count && ok; start += SM_KEYS, ++n) {
                if (start == 0) { ok = mbar_wait_warp(&q_full, row_n & 1); ++row_n; }
                for (int j = 0; j < 5 && ok; ++j) {
                    if (!mbar_wait_warp(k_full + j, n & 1)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        for (int b = 2 * j; b < min(2 * j + 2, SM_BOXES); ++b)
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                umma_bf16(tmem, umma_desc_sw128(k_addr + b * SM_KBOX + k * 32), umma_desc_sw128(q_addr + b * SM_QBOX + k * 32), idesc_s,
                                          (b > 0 || k > 0) ? 1u : 0u);
                        if (j == 4) umma_commit(&s_full);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (!mbar_wait_warp(&p_full, n & 1)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int steps = (min(SM_KEYS, count - start) + 15) >> 4;
                if (elect_one()) {
                    for (int j = 0; j < 4; ++j) {
                        for (int k = 0; k < steps; ++k)
                            umma_bf16(tmem + 64 + j * 64, sm_desc_mn(k_addr + 2 * j * SM_KBOX + k * 2048), sm_desc_mn(p_addr + k * 2048), idesc_o,
                                      (start > 0 || k > 0) ? 1u : 0u);
                        umma_commit(o_done + j);
                    }
                }
                __syncwarp();
            }
        }
    } else {
        // ---- softmax: warps w and w + 4 share the keys of TMEM lanes 32 w .., the first with heads 0-31, the second with 32-63 -------
        const int half = warp >> 2, key = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, s_addr = tmem + lanes + half * SM_HALF, o_addr = tmem + lanes + 64 + half * SM_HALF;
        const float scale2 = a.scale * SM_LOG2E;
        unsigned char* p_row = p_s + (key >> 3) * 1024 + (key & 7) * 128;
        float *ref = ref_s[warp], *fix = fix_s[warp];
        bool ok = true;  // after a wait that ran out: meaningless from there on, nothing is waited for or stored, but every barrier is still met
        for (int i = blockIdx.x; i < a.rows; i += gridDim.x) {
            const int r = a.rows - 1 - i, count = keys_of(r);
            bf16* out = a.o_lat + ((int64_t)r * SM_H + half * SM_HALF) * SM_L;
            if (count == 0) {  // no selected key: zeros
                for (int v = threadIdx.x & 127; v < SM_HALF * SM_L / 8; v += 128) reinterpret_cast<uint4*>(out)[v] = make_uint4(0, 0, 0, 0);
                continue;
            }
            float l[SM_HALF], run = -INFINITY, odd = 0.f;  // run: reference of head `lane` of the half
#pragma unroll
            for (int h = 0; h < SM_HALF; ++h) l[h] = 0.f;
            for (int start = 0; start < count; start += SM_KEYS, ++n) {
                const bool live = key < count - start;
                if (ok) ok = mbar_wait_warp(&s_full, n & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float s[SM_HALF];
                sm_ld32(s_addr, s);
                // the maximum of the warp's keys per head: halves of the heads change sides until lane h has head h
                float top[SM_HALF];
#pragma unroll
                for (int h = 0; h < SM_HALF; ++h) top[h] = live ? s[h] * scale2 : -INFINITY;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int h = 0; h < 16; ++h)
                        if (h < o) {
                            const bool up = lane & o;
                            const float keep = up ? top[h + o] : top[h], send = up ? top[h] : top[h + o];
                            top[h] = fmaxf(keep, __shfl_xor_sync(0xffffffffu, send, o));
                        }
                top_s[warp][lane] = top[0];
                sm_barrier();  // (nobody writes the next block's before all have given up this block's weights)
                const float (*tops)[SM_HALF] = top_s + half * 4;
                const float next = fmaxf(run, fmaxf(fmaxf(tops[0][lane], tops[1][lane]), fmaxf(tops[2][lane], tops[3][lane])));
                const float factor = next == -INFINITY ? 1.f : sm_exp2(run - next);
                fix[lane] = factor;
                ref[lane] = next == -INFINITY ? 0.f : next;
                run = next;
                __syncwarp();
                if (lane == 0 && (warp & 3) == 0) mbar_arrive(&fix_full);  // the products of the block before are complete: the scores of this one follow them
                if (__any_sync(0xffffffffu, factor != 1.f) && start > 0)
#pragma unroll
                    for (int h = 0; h < SM_HALF; ++h) l[h] *= fix[h];
#pragma unroll
                for (int c = 0; c < SM_HALF; c += 8) {
                    const float4 m0 = *reinterpret_cast<const float4*>(ref + c), m1 = *reinterpret_cast<const float4*>(ref + c + 4);
                    const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
                    float p[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        odd = live ? fmaf(s[c + e], 0.f, odd) : odd;  // NaN if a score is not finite
                        p[e] = live ? sm_exp2(fmaf(s[c + e], scale2, -m[e])) : 0.f;
                        l[c + e] += p[e];
                    }
                    *reinterpret_cast<uint4*>(p_row + (((half * 4 + (c >> 3)) ^ (key & 7)) << 4)) =
                        make_uint4(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]), pack_bf16(p[4], p[5]), pack_bf16(p[6], p[7]));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full);
            }
            if (ok && odd != 0.f) raise_status(a.status, GLMB_STATUS_NONFINITE);
            // sums over the keys: halves of the heads change sides until lane h has head h
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < 16; ++h)
                    if (h < o) {
                        const bool up = lane & o;
                        const float keep = up ? l[h + o] : l[h], send = up ? l[h] : l[h + o];
                        l[h] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
            sum_s[warp][lane] = l[0];
            sm_barrier();
            const float (*sums)[SM_HALF] = sum_s + half * 4;
            // (in arrays of this warp that nobody else reads: `fix` may still be in use, and the sums are)
            const float total = (sums[0][lane] + sums[1][lane]) + (sums[2][lane] + sums[3][lane]);
            float *const all = ref, *const inv = inv_s[warp];
            all[lane] = total;
            inv[lane] = __frcp_rn(total);
            __syncwarp();
            if (ok) ok = mbar_wait_warp(o_done + 3, (n - 1) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {  // 128 latent columns at a time; a lane has one of them
                float o[32];
                sm_ld32(o_addr + c * 64, o);
                const int at = c * 128 + (warp & 3) * 32 + (lane & ~1);
#pragma unroll
                for (int e = 0; e < 32; e += 2) {  // neighbours swap, so that each stores two columns of one head
                    const float x = sm_quotient(o[e], all[e], inv[e]), y = sm_quotient(o[e + 1], all[e + 1], inv[e + 1]);
                    const float got = __shfl_xor_sync(0xffffffffu, (lane & 1) ? x : y, 1);
                    if (ok) *reinterpret_cast<uint32_t*>(out + (e + (lane & 1)) * SM_L + at) = (lane & 1) ? pack_bf16(got, y) : pack_bf16(x, got);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            sm_barrier();  // what the warps share has been read
        }
        if (!ok && lane == 0) raise_status(a.status, GLMB_STATUS_WAIT_TIMEOUT);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 12) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// The shapes and alignments this kernel takes (TMA on the queries, 16-byte copies of the cache rows, vector stores).
bool sparse_mla_tc_takes(const void* q_full, const void* kv_cache, const void* o_lat, int H, int L, int rd) {
    return H == SM_H && L == SM_L && rd == SM_W - SM_L &&
           !((reinterpret_cast<uintptr_t>(q_full) | reinterpret_cast<uintptr_t>(kv_cache) | reinterpret_cast<uintptr_t>(o_lat)) & 15);
}

int launch_sparse_mla_tc(const void* q_full, const void* kv_cache, const int* sel_local, const int* sel_counts, const int* row_lane, int rows,
                         int layer, int layers, int local_cap, int top_k, float scale, void* o_lat, uint32_t* status, cudaStream_t stream) {
    CUtensorMap map_q;
    if (make_map(&map_q, q_full, (uint64_t)rows * SM_H, SM_W, SM_W, SM_H)) return 3;
    static DeviceOnce once;
    const int dev = once.pending();
    if (dev != DeviceOnce::SET) {
        const cudaError_t e = cudaFuncSetAttribute(sparse_mla_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_SMEM);
        if (e != cudaSuccess) return (int)e;
        once.mark(dev);
    }
    SparseMlaArgs a;
    a.kv_cache = (const bf16*)kv_cache; a.sel_local = sel_local; a.sel_counts = sel_counts; a.row_lane = row_lane; a.o_lat = (bf16*)o_lat;
    a.rows = rows; a.layer = layer; a.layers = layers; a.local_cap = local_cap; a.top_k = top_k; a.scale = scale; a.status = status;
    GLMB_LAUNCH(sparse_mla_tc_kernel, rows < 148 ? rows : 148, SM_THREADS, SM_SMEM, stream, map_q, a);
    return (int)cudaGetLastError();
}

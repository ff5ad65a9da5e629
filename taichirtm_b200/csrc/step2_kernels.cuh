// Two time steps per launch (temporal blocking) of the fused elastic step.
//
// step2_kernel advances every shot by steps A (time p.it) and B (time p.it2)
// in one pass over the wavefield: the state is read once (before A) and
// written once (after B), the material once, so a launch costs the HBM
// traffic of one single step for two steps of work.  Every cell's
// arithmetic is the single-step kernel's, operation by operation, so the
// result is bit-identical to two launches of step_kernel.
//
// Dependencies.  One step reaches one row and one column in each direction:
// forward, the velocity of row i reads the stress of rows i-1, i and the
// stress of row i reads the new velocity of rows i, i+1; backward the other
// way round (backward_modeling.py:312-380).  A warp streaming down rows k
// therefore runs four row updates per iteration:
//   forward:  A velocity k, A stress k-1, B velocity k-1, B stress k-2
//   backward: A velocity k-1, A stress k-1, B velocity k-2, B stress k-2
// and a task that writes rows [ia, ib) recomputes step A on one extra row
// above and below (rows ia-1 .. ib) from the old state of rows ia-2 .. ib+1.
// Row indices are clamped to the pad rows -1 .. nx of the shot block: rows -2
// and nx+1 read the zero pad state (no update touches a non-interior cell, so
// pad rows stay zero), and the material read there feeds only updates of
// non-interior cells, which the interior selects discard.  The loads need no
// per-row branch.
//
// Columns.  Lanes 0 and 31 carry VEC halo columns.  After step A only their
// outermost column is wrong (its neighbour is outside the warp); after step
// B the two outermost ones.  With VEC >= 2 every column that an owner lane
// (1..30) reads is still exact, so the single-step decomposition is kept.
//
// Epilogues.  Step A's values are recorded (forward receivers,
// _record_seismogram_kernel), snapshotted (forward) or correlated (backward
// imaging) for rows [ia, ib) exactly like a single step; they are not
// written back.  The finite check runs on step B only: the host never pairs
// a step that is checked as step A, so a shot that fails stops at the step
// where the reference stops.
#pragma once
#include <type_traits>

#include "f32x2.cuh"
#include "step_kernels.cuh"

namespace rtm {

// A lane's VEC columns of one row, as VEC / 2 packed pairs (f32x2.cuh).
template <int VEC>
struct SigRow { f2 xx[VEC / 2], zz[VEC / 2], xz[VEC / 2], yx[VEC / 2], yz[VEC / 2]; };
template <int VEC>
struct VelRow { f2 u[VEC / 2], w[VEC / 2], v[VEC / 2]; };
template <int VEC>
struct MatRow { f2 lam[VEC / 2], mu[VEC / 2], mxz[VEC / 2], myx[VEC / 2], myz[VEC / 2], sm[VEC / 2]; };

template <int N>
__device__ __forceinline__ void zero_arr(f2 (&a)[N]) {
#pragma unroll
    for (int q = 0; q < N; ++q) a[q] = 0ull;
}

template <int N>
__device__ __forceinline__ void copy_arr(f2 (&d)[N], const f2 (&s)[N]) {
#pragma unroll
    for (int q = 0; q < N; ++q) d[q] = s[q];
}

// Vector loads and stores of VEC / 2 pairs.
template <int N>
__device__ __forceinline__ void ldp(f2 (&v)[N], const float *__restrict__ p) {
    if constexpr (N == 2) {
        const ulonglong2 t = ldg_chk(reinterpret_cast<const ulonglong2 *>(p));
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = ldg_chk(reinterpret_cast<const f2 *>(p));
    }
}
template <int N>
__device__ __forceinline__ void stp(float *__restrict__ p, const f2 (&v)[N]) {
    if (!RTM_DBG_OK(p, N * sizeof(f2))) return;
    if constexpr (N == 2) *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v[0], v[1]);
    else *reinterpret_cast<f2 *>(p) = v[0];
}
template <int N>
__device__ __forceinline__ void unpack(float (&d)[2 * N], const f2 (&s)[N]) {
#pragma unroll
    for (int q = 0; q < N; ++q) { d[2 * q] = f2_lo(s[q]); d[2 * q + 1] = f2_hi(s[q]); }
}
// Differences with the next lower / higher column; nb: the neighbouring lane's.
template <class A, int N>
__device__ __forceinline__ f2 diff_lo(const f2 (&x)[N], int q, float nb) {
    return A::pack(f2_lo(x[q]) - (q > 0 ? f2_hi(x[q > 0 ? q - 1 : 0]) : nb), f2_hi(x[q]) - f2_lo(x[q]));
}
template <class A, int N>
__device__ __forceinline__ f2 diff_hi(const f2 (&x)[N], int q, float nb) {
    return A::pack(f2_hi(x[q]) - f2_lo(x[q]), (q < N - 1 ? f2_lo(x[q < N - 1 ? q + 1 : 0]) : nb) - f2_hi(x[q]));
}

// Plain (coherent) vector load for the Kahan image: one thread may read a
// cell again after writing it in the same launch (steps A and B both
// imaging), which the read-only path (ld.global.nc) does not allow.
template <int VEC>
__device__ __forceinline__ void ldv_coherent(float (&v)[VEC], float *p) {
    if (!RTM_DBG_OK(p, VEC * sizeof(float))) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) v[q] = 0.f;
        return;
    }
    if constexpr (VEC == 4) {
        const float4 t = *reinterpret_cast<float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VEC == 2) {
        const float2 t = *reinterpret_cast<float2 *>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = *p;
    }
}

// Material ring (RING = true): the material and inverse-density rows reach a
// warp through a per-warp shared-memory ring of RING2_ROWS rows, filled by
// cp.async one iteration ahead, instead of rolling through registers.  Each
// lane copies and reads back only its own VEC columns, so its own
// wait_group is the only synchronisation.  It frees about 30 registers per
// thread, i.e. more resident warps.  Fields per ring row: P-SV lam, mu, mxz,
// 1/rho_u, 1/rho_w; SH myx, myz, 1/rho; the surface mask.
constexpr int RING2_ROWS = 4;
template <int MODE>
__host__ __device__ constexpr int ring2_fields() { return ((MODE & 1) ? 5 : 0) + ((MODE & 2) ? 3 : 0); }
// State ring (SR, forward with RING): the state rows come through a ring of their
// own, three rows deep: two rows ahead instead of one, and 20 registers (vec 4)
// fewer copies per row.  launch_step2 takes it where the rings leave nearly as
// many warps on an SM (64 shots of 801 columns, vec 4: 166.4 -> 183.7 Gcell/s);
// elsewhere the state rolls through registers.  Backward launches gain nothing
// from it (154.6 -> 156.7, and 14 shots lose: 128 -> 125).
template <bool SR>
__host__ __device__ constexpr int ring2_state_rows() { return SR ? 3 : 0; }
template <bool SR, int MODE, int VEC>
__host__ __device__ constexpr size_t ring2_smem_per_warp(bool surface) {
    return ((size_t)RING2_ROWS * (ring2_fields<MODE>() + (surface ? 1 : 0)) + ring2_state_rows<SR>() * ring2_fields<MODE>()) * 32 * VEC * sizeof(float);
}

// Packed arithmetic, or scalar?  Scalar against packed, 0.2 to 7.7 million cells:
// without the rings 0.94 to 1.0 with vec 2 (its two columns are one chain of packed
// operations where they were two; launch_step2_as has the exception), 1.0 to 1.04 for
// P-SV and SH with vec 4.  With the material
// ring and the state in registers 0.92 to 1.0 for P-SV with vec 2 and for SH, 1.0
// to 1.1 for the rest; with the state ring 1.0 to 1.1.  Backward with the ring 0.96
// to 1.0 for SH with vec 2, else 0.95 to 1.15 either way.
__host__ __device__ constexpr bool step2_packed(int dir, int mode, int vec, bool ring, bool state_ring) {
    if (!ring) return vec == 4 && mode != 3;
    if (dir == 1) return mode != 2 || vec == 4;
    return state_ring || mode == 3 || (mode == 1 && vec == 4);
}
// CTAs per SM that the register budget is cut for (0: as it comes).  Both wave types
// backward, vec 2, 8 warps: 140 registers left one CTA on an SM.  SH, vec 2, 4 warps,
// no ring: 100 to 120 registers left four CTAs where 96, without spills, leave five.
__host__ __device__ constexpr int step2_min_ctas(int dir, int mode, int vec, bool ring, bool uni, int warps) {
    if (mode == 3 && vec == 2 && ring && !uni && dir == 1) return 2;
    return mode == 2 && vec == 2 && !ring && warps == 4 ? 5 : 0;
}

// STOREA: also store step A's state (rows [ia, ib), into p.souta), for the
// forward recompute of the FWI adjoint, which needs the state after every step.
// CKPT: step B's state is also stored, block-scaled to 16 bits, into the
// checkpoint slot p.ck (ckpt_pack.cuh); forward P-SV only.
// WARPS: the most warps a CTA is launched with.
// UNI: launched with one warp per CTA, the task is blockIdx.x.  Everything
// derived from the task (shot, strip, row range, loop bounds, fast-path
// choices) is then provably the same for the whole warp, so the compiler
// keeps it in uniform registers and branches on it without divergence
// bookkeeping; the arithmetic of every cell is unchanged.
template <int DIR, int MODE, int VEC, bool RING = false, bool STOREA = false, bool CKPT = false, bool UNI = false, bool SR = false, int WARPS = 8,
          bool PACKED = step2_packed(DIR, MODE, VEC, RING, SR)>
__global__ void __launch_bounds__(UNI ? 32 : 32 * WARPS, step2_min_ctas(DIR, MODE, VEC, RING, UNI, WARPS)) step2_kernel(const StepParams p) {
    static_assert(VEC >= 2, "two steps per launch need two halo columns per side");
    static_assert(!STOREA || DIR == 0, "only the forward recompute stores step A");
    static_assert(!SR || (DIR == 0 && RING), "the state ring is the forward kernel's");
    static_assert(!CKPT || (DIR == 0 && MODE == 1), "checkpoint stores are forward P-SV");
    constexpr bool PSV = (MODE & 1) != 0;
    constexpr bool SH = (MODE & 2) != 0;
    constexpr int W = 30 * VEC;
    using A = Pairs<PACKED>;
    using Sig = SigRow<VEC>;
    using Vel = VelRow<VEC>;
    using Mat = MatRow<VEC>;
    const int lane = threadIdx.x & 31;
    const int task = UNI ? (int)blockIdx.x : (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (task >= p.n_work) return;
    const int4 wk = p.work[task];
    if (shot_stopped(p, wk.x)) return;
    const ShotDev sh = p.shots[wk.x];
    const int nx = sh.nx, nz = p.nz, P = p.pitch;
    const int j0 = (wk.y & 0xFFFFF) * W;
    const bool no_src = (wk.y >> 20) & 1, no_rec = (wk.y >> 21) & 1;
    const int c0 = j0 - VEC + VEC * lane;
    const bool owner = lane >= 1 && lane <= 30;
    const int ia = wk.z, ib = wk.w;
    // The fast paths are chosen per warp (one uniform branch): a warp whose
    // columns are not all interior / outside the sponge runs the general path
    // on every lane instead of both paths.
    const bool strip_in = __all_sync(FULL, c0 >= 1 && c0 + VEC - 1 <= nz - 2);
    const bool strip_far = __all_sync(FULL, nz - 1 - (c0 + VEC - 1) >= p.fw);
    auto all_in = [&](int i) { return strip_in && i >= 1 && i <= nx - 2; };
    auto all_far = [&](int i) { return strip_far && i >= p.fw && nx - 1 - i >= p.fw; };
    // The general path's per-cell interior test and sponge coefficient,
    // factored into a column part fixed for the task (here, once per lane)
    // and a warp-uniform row part (ColRow below): the same cells are interior
    // and the same sponge entry is chosen as by interior() and sponge_coef().
    bool col_sp[VEC];
    unsigned col_m[VEC];  // all ones for an interior column
    int col_db[VEC];
    float col_cr[VEC];
#pragma unroll
    for (int q = 0; q < VEC; ++q) {
        const int j = c0 + q;
        col_m[q] = (unsigned)(j - 1) < (unsigned)(nz - 2) ? ~0u : 0u;
        col_db[q] = nz - 1 - j;  // distance to the bottom edge
        col_sp[q] = col_db[q] >= 0 && col_db[q] < p.fw;
        col_cr[q] = col_sp[q] ? ldg_chk(p.sponge + col_db[q]) : 1.0f;
    }
    const long long soff = sh.state_off + (long long)(c0 + COL_OFF);
    const long long moff = (long long)sh.x0 * P + (long long)(c0 + COL_OFF);
    const float dt = p.dt, idx = p.inv_dx, idz = p.inv_dz;
    const f2 dt2 = A::pack(dt, dt), idx2 = A::pack(idx, idx), idz2 = A::pack(idz, idz), nz2 = A::pack(p.neg_zero, p.neg_zero);
    constexpr int NP = VEC / 2;
    // CKPT: scale block of row -1 of this task's strip (padded row 0 of the shot)
    long long ck_blk0 = 0;
    if constexpr (CKPT) ck_blk0 = (sh.state_off / P) * p.ck.nblk + (wk.y & 0xFFFFF) * (W / ckpt_block_cols(VEC));
    // rows -1 and nx are the zero pad rows of the shot block (and of the
    // material window); rows beyond them read the pad row (header comment)
    auto rowc = [&](int i) { return min(max(i, -1), nx); };
    auto LSt = [&](f2 (&v)[NP], int f, int i) { ldp<NP>(v, p.sin[f] + soff + (long long)(rowc(i) + 1) * P); };
    auto LMt = [&](f2 (&v)[NP], int m, int i) { ldp<NP>(v, p.mat[m] + moff + (long long)(rowc(i) + 1) * P); };
    auto load_sig = [&](int i, Sig &s) {
        if constexpr (PSV) { LSt(s.xx, F_SXX, i); LSt(s.zz, F_SZZ, i); LSt(s.xz, F_SXZ, i); }
        if constexpr (SH) { LSt(s.yx, F_SYX, i); LSt(s.yz, F_SYZ, i); }
    };
    auto load_vel = [&](int i, Vel &v) {
        if constexpr (PSV) { LSt(v.u, F_U, i); LSt(v.w, F_W, i); }
        if constexpr (SH) LSt(v.v, F_V, i);
    };
    auto load_ir = [&](int i, Vel &v) {
        if constexpr (PSV) { LMt(v.u, M_IRU, i); LMt(v.w, M_IRW, i); }
        if constexpr (SH) LMt(v.v, M_IR, i);
    };
    auto load_mat = [&](int i, Mat &m) {
        if constexpr (PSV) { LMt(m.lam, M_LAM, i); LMt(m.mu, M_MU, i); LMt(m.mxz, M_MXZ, i); }
        if constexpr (SH) { LMt(m.myx, M_MYX, i); LMt(m.myz, M_MYZ, i); }
        if (p.surface) {
            ldp<NP>(m.sm, p.surface + moff + (long long)(rowc(i) + 1) * P);
        } else {
#pragma unroll
            for (int q = 0; q < NP; ++q) m.sm[q] = A::pack(1.f, 1.f);
        }
    };
    // ---- material ring (RING): slot of a row, copy-in, read-back
    constexpr int NRF = ring2_fields<MODE>();
    constexpr int RF_LAM = 0, RF_MU = 1, RF_MXZ = 2, RF_IRU = 3, RF_IRW = 4;
    constexpr int RF_MYX = PSV ? 5 : 0, RF_MYZ = RF_MYX + 1, RF_IR = RF_MYX + 2;
    constexpr int RF_SM = NRF;
    const int nrf = NRF + (p.surface ? 1 : 0);  // the surface mask's rows only where there is one
    extern __shared__ float step2_smem[];
    static_assert((RING2_ROWS & (RING2_ROWS - 1)) == 0, "the ring slot is the row modulo a power of two");
    // this lane's VEC floats of slot 0, field 0; a (slot, field) is a fixed
    // 32-bit offset from it (rows >= -2: row & (RING2_ROWS - 1) is the slot)
    float *const ring = step2_smem + (UNI ? 0 : (int)(threadIdx.x >> 5) * ((RING2_ROWS * nrf + ring2_state_rows<SR>() * NRF) * 32 * VEC)) + lane * VEC;
    float *const sring = ring + RING2_ROWS * nrf * (32 * VEC);
    auto rslot = [&](int row, int f) { return ring + ((row & (RING2_ROWS - 1)) * nrf + f) * (32 * VEC); };
    // state ring: slot 0, 1, 2 of the rows in turn; fields as NFIELD of the modes
    auto sslot = [&](int slot, int f) { return sring + (slot * NRF + f) * (32 * VEC); };
    // stress and velocity of a row into a slot
    auto state_issue = [&](int slot, int row) {
        if (row <= ib + 1) {
            auto put = [&](int f, int field, int r) {
                cp_async_vec<VEC>(sslot(slot, f), p.sin[field] + soff + (long long)(rowc(r) + 1) * P);
            };
            constexpr int o = PSV ? 5 : 0;
            if constexpr (PSV) {
                put(0, F_SXX, row); put(1, F_SZZ, row); put(2, F_SXZ, row);
                put(3, F_U, row); put(4, F_W, row);
            }
            if constexpr (SH) { put(o, F_SYX, row); put(o + 1, F_SYZ, row); put(o + 2, F_V, row); }
        }
        cp_async_commit();
    };
    auto rd_state = [&](int slot, Sig &sg, Vel &v) {
        auto get = [&](int f, f2 (&x)[NP]) {
            const float *a = sslot(slot, f);
            if constexpr (NP == 2) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(a);
                x[0] = t.x; x[1] = t.y;
            } else {
                x[0] = *reinterpret_cast<const f2 *>(a);
            }
        };
        constexpr int o = PSV ? 5 : 0;
        if constexpr (PSV) { get(0, sg.xx); get(1, sg.zz); get(2, sg.xz); get(3, v.u); get(4, v.w); }
        if constexpr (SH) { get(o, sg.yx); get(o + 1, sg.yz); get(o + 2, v.v); }
    };
    (void)state_issue; (void)rd_state;
    auto ring_issue = [&](int row) {
        auto put = [&](int f, const float *src) {
            cp_async_vec<VEC>(rslot(row, f), src + moff + (long long)(rowc(row) + 1) * P);
        };
        if constexpr (PSV) {
            put(RF_LAM, p.mat[M_LAM]); put(RF_MU, p.mat[M_MU]); put(RF_MXZ, p.mat[M_MXZ]);
            put(RF_IRU, p.mat[M_IRU]); put(RF_IRW, p.mat[M_IRW]);
        }
        if constexpr (SH) { put(RF_MYX, p.mat[M_MYX]); put(RF_MYZ, p.mat[M_MYZ]); put(RF_IR, p.mat[M_IR]); }
        if (p.surface) put(RF_SM, p.surface);
        cp_async_commit();  // one group per issued row, so the group counts stay aligned
    };
    auto rd_ring = [&](int row, int f, f2 (&v)[NP]) {
        const float *s = rslot(row, f);
        if constexpr (NP == 2) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(s);
            v[0] = t.x; v[1] = t.y;
        } else {
            v[0] = *reinterpret_cast<const f2 *>(s);
        }
    };
    auto ring_ir = [&](int row, Vel &v) {
        if constexpr (PSV) { rd_ring(row, RF_IRU, v.u); rd_ring(row, RF_IRW, v.w); }
        if constexpr (SH) rd_ring(row, RF_IR, v.v);
    };
    auto ring_mat = [&](int row, Mat &m) {
        if constexpr (PSV) { rd_ring(row, RF_LAM, m.lam); rd_ring(row, RF_MU, m.mu); rd_ring(row, RF_MXZ, m.mxz); }
        if constexpr (SH) { rd_ring(row, RF_MYX, m.myx); rd_ring(row, RF_MYZ, m.myz); }
        if (p.surface) {
            rd_ring(row, RF_SM, m.sm);
        } else {
#pragma unroll
            for (int q = 0; q < NP; ++q) m.sm[q] = A::pack(1.f, 1.f);
        }
    };
    (void)ring_issue; (void)ring_ir; (void)ring_mat;

    auto cp_sig = [&](Sig &d, const Sig &s) {
        if constexpr (PSV) { copy_arr<NP>(d.xx, s.xx); copy_arr<NP>(d.zz, s.zz); copy_arr<NP>(d.xz, s.xz); }
        if constexpr (SH) { copy_arr<NP>(d.yx, s.yx); copy_arr<NP>(d.yz, s.yz); }
    };
    auto cp_vel = [&](Vel &d, const Vel &s) {
        if constexpr (PSV) { copy_arr<NP>(d.u, s.u); copy_arr<NP>(d.w, s.w); }
        if constexpr (SH) copy_arr<NP>(d.v, s.v);
    };
    auto cp_mat = [&](Mat &d, const Mat &s) {
        if constexpr (PSV) { copy_arr<NP>(d.lam, s.lam); copy_arr<NP>(d.mu, s.mu); copy_arr<NP>(d.mxz, s.mxz); }
        if constexpr (SH) { copy_arr<NP>(d.myx, s.myx); copy_arr<NP>(d.myz, s.myz); }
        copy_arr<NP>(d.sm, s.sm);
    };
    auto zero_sig = [&](Sig &s) {
        if constexpr (PSV) { zero_arr<NP>(s.xx); zero_arr<NP>(s.zz); zero_arr<NP>(s.xz); }
        if constexpr (SH) { zero_arr<NP>(s.yx); zero_arr<NP>(s.yz); }
    };
    auto zero_vel = [&](Vel &v) {
        if constexpr (PSV) { zero_arr<NP>(v.u); zero_arr<NP>(v.w); }
        if constexpr (SH) zero_arr<NP>(v.v);
    };

    // Velocity update of row r (step time t), the arithmetic of step_kernel.
    // Forward: sc = stress row r, sp = row r-1.  Backward: sc = row r+1,
    // sp = row r.  vo = velocity of row r before the update.  FAST (every
    // column of the lane interior) drops the interior select, nothing else.
    // Edge cells keep their value: their increment is cleared bitwise, so not
    // even a NaN of a failing shot gets in.
    auto clip = [&](f2 d, int q, unsigned rm) -> f2 {
        return (f2)((unsigned)(d >> 32) & col_m[2 * q + 1] & rm) << 32 | ((unsigned)d & col_m[2 * q] & rm);
    };
    auto vel_cells = [&](auto fast_tag, int r, const Sig &sc, const Sig &sp, const Vel &vo, const Vel &ir,
                         Vel &out, float zz_nb, float xz_nb, float yz_nb) {
        constexpr bool FAST = decltype(fast_tag)::value;
        unsigned rm = ~0u;
        if constexpr (!FAST) rm = (unsigned)(r - 1) < (unsigned)(nx - 2) ? ~0u : 0u;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            if constexpr (PSV) {
                const f2 sxx_x = A::mul(A::sub(sc.xx[q], sp.xx[q]), idx2, nz2);  // fm:332, bm:333
                const f2 sxz_x = A::mul(A::sub(sc.xz[q], sp.xz[q]), idx2, nz2);  // fm:334, bm:335
                f2 dzz, dxz;
                if constexpr (DIR == 0) { dzz = diff_lo<A>(sc.zz, q, zz_nb); dxz = diff_lo<A>(sc.xz, q, xz_nb); }
                else { dzz = diff_hi<A>(sp.zz, q, zz_nb); dxz = diff_hi<A>(sp.xz, q, xz_nb); }
                const f2 szz_z = A::mul(dzz, idz2, nz2);                          // fm:333, bm:334
                const f2 sxz_z = A::mul(dxz, idz2, nz2);                          // fm:335, bm:336
                f2 du = A::mul(A::mul(A::add(sxx_x, sxz_z), dt2, nz2), ir.u[q], nz2);  // fm:339, bm:340 (negated)
                f2 dw = A::mul(A::mul(A::add(sxz_x, szz_z), dt2, nz2), ir.w[q], nz2);  // fm:340, bm:341
                if constexpr (!FAST) { du = clip(du, q, rm); dw = clip(dw, q, rm); }
                out.u[q] = DIR == 0 ? A::add(vo.u[q], du) : A::sub(vo.u[q], du);
                out.w[q] = DIR == 0 ? A::add(vo.w[q], dw) : A::sub(vo.w[q], dw);
            }
            if constexpr (SH) {
                const f2 syx_x = A::mul(A::sub(sc.yx[q], sp.yx[q]), idx2, nz2);  // fm:343, bm:343
                f2 dyz;
                if constexpr (DIR == 0) dyz = diff_lo<A>(sc.yz, q, yz_nb);
                else dyz = diff_hi<A>(sp.yz, q, yz_nb);
                const f2 syz_z = A::mul(dyz, idz2, nz2);                          // fm:344, bm:344
                f2 dv = A::mul(A::mul(A::add(syx_x, syz_z), dt2, nz2), ir.v[q], nz2);  // fm:347, bm:345
                if constexpr (!FAST) dv = clip(dv, q, rm);
                out.v[q] = DIR == 0 ? A::add(vo.v[q], dv) : A::sub(vo.v[q], dv);
            }
        }
    };
    auto vel_update = [&](int r, int t, const Sig &sc, const Sig &sp, const Vel &vo, const Vel &ir, Vel &out) {
        // column neighbour: j-1 of row r (forward), j+1 of row r (backward)
        float zz_nb = 0.f, xz_nb = 0.f, yz_nb = 0.f;
        if constexpr (DIR == 0) {
            if constexpr (PSV) {
                zz_nb = __shfl_up_sync(FULL, f2_hi(sc.zz[NP - 1]), 1);
                xz_nb = __shfl_up_sync(FULL, f2_hi(sc.xz[NP - 1]), 1);
            }
            if constexpr (SH) yz_nb = __shfl_up_sync(FULL, f2_hi(sc.yz[NP - 1]), 1);
        } else {
            if constexpr (PSV) {
                zz_nb = __shfl_down_sync(FULL, f2_lo(sp.zz[0]), 1);
                xz_nb = __shfl_down_sync(FULL, f2_lo(sp.xz[0]), 1);
            }
            if constexpr (SH) yz_nb = __shfl_down_sync(FULL, f2_lo(sp.yz[0]), 1);
        }
        if (all_in(r)) vel_cells(std::true_type{}, r, sc, sp, vo, ir, out, zz_nb, xz_nb, yz_nb);
        else vel_cells(std::false_type{}, r, sc, sp, vo, ir, out, zz_nb, xz_nb, yz_nb);
        // point injection at time t: forward sources (fm:421-443), backward
        // observed data (bm:452-460); halo lanes too, so halo cells are exact
        if (r < 0 || r >= nx) return;
        if constexpr (DIR == 0) {
            if (no_src) return;
            const int e0 = ldg_chk(p.src_ptr + sh.src_row0 + r), e1 = ldg_chk(p.src_ptr + sh.src_row0 + r + 1);
            for (int e = e0; e < e1; ++e) {
                const int2 en = ldg_chk(p.src_ent + e);
                const int q = en.x - c0;
                if (q < 0 || q >= VEC) continue;
                const bool in = interior(r, en.x, nx, nz);
                const float f = p.src_factor;
                const size_t ti = (size_t)en.y * p.nt + t;
                auto add = [&](f2 (&x)[NP], const f2 (&ir2)[NP], const float *wav, bool masked) {
                    const float wf = ldg_chk(wav + ti) * f;
#pragma unroll
                    for (int k = 0; k < NP; ++k) {  // x + -0.0 is x: the other columns take part
                        const float b = q & 1 ? f2_hi(ir2[k]) : f2_lo(ir2[k]);
                        const float a = wf * (in || !masked ? b : __int_as_float(0x7f800000));
                        x[k] = A::add(x[k], A::pack(q == 2 * k ? a : -0.0f, q == 2 * k + 1 ? a : -0.0f));
                    }
                };
                if constexpr (PSV) { add(out.u, ir.u, p.wav[0], true); add(out.w, ir.w, p.wav[2], true); }
                if constexpr (SH) add(out.v, ir.v, p.wav[1], false);
            }
        } else {
            if (no_rec) return;
            const int e0 = ldg_chk(p.rec_ptr + sh.rec_row0 + r), e1 = ldg_chk(p.rec_ptr + sh.rec_row0 + r + 1);
            for (int e = e0; e < e1; ++e) {
                const int2 en = ldg_chk(p.rec_ent + e);
                const int q = en.x - c0;
                if (q < 0 || q >= VEC) continue;
                const size_t ti = (size_t)t * p.nrec_total + en.y;
                auto add = [&](f2 (&x)[NP], const float *obs) {
                    const float a = ldg_chk(obs + ti);
#pragma unroll
                    for (int k = 0; k < NP; ++k)
                        x[k] = A::add(x[k], A::pack(q == 2 * k ? a : -0.0f, q == 2 * k + 1 ? a : -0.0f));
                };
                if constexpr (PSV) { add(out.u, p.obs[0]); add(out.w, p.obs[2]); }
                if constexpr (SH) add(out.v, p.obs[1]);
            }
        }
    };

    // Stress update of row r, then absorbing and the surface mask of the
    // next step: va = new velocity of row r, vb = of row r+1 (forward) or
    // r-1 (backward), base = stress of row r before the step.  FAST (every
    // column of the lane interior, outside the sponge, no topography mask)
    // drops the interior select and the multiplications by a coefficient of
    // exactly 1.0, which leave every value unchanged.
    auto stress_cells = [&](auto fast_tag, int r, const Vel &va, const Vel &vb, const Sig &base, const Mat &m,
                            Sig &os, Vel &ov, float nu, float nw, float nv) {
        constexpr bool FAST = decltype(fast_tag)::value;
        // row part of the sponge choice (sponge_coef): d = r if the row is in
        // the left sponge and the cell is farther from the bottom, d = nx-1-r
        // likewise for the right sponge, d = the bottom distance if that is
        // in the sponge and no larger than both row distances (last wins)
        bool ra = false, rb = false;
        unsigned rm = ~0u;
        int dr = 0;
        float cr_i = 1.0f, cr_dr = 1.0f;
        if constexpr (!FAST) {
            rm = (unsigned)(r - 1) < (unsigned)(nx - 2) ? ~0u : 0u;
            dr = nx - 1 - r;
            ra = r >= 0 && r < p.fw;
            rb = dr >= 0 && dr < p.fw;
            if (ra) cr_i = ldg_chk(p.sponge + r);
            if (rb) cr_dr = ldg_chk(p.sponge + dr);
        }
        const f2 sdt2 = DIR == 0 ? dt2 : A::pack(-dt, -dt);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            f2 c = 0ull;
            if constexpr (!FAST) {
                float cr[2] = {1.0f, 1.0f};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = 2 * q + h;
                    if (ra && col_db[k] > r) cr[h] = cr_i;
                    if (rb && col_db[k] > dr) cr[h] = cr_dr;
                    if (col_sp[k] && r >= col_db[k] && dr >= col_db[k]) cr[h] = col_cr[k];
                }
                c = A::pack(cr[0], cr[1]);
            }
            if constexpr (PSV) {
                f2 dux, dwx, duz, dwz;
                if constexpr (DIR == 0) {
                    dux = A::sub(vb.u[q], va.u[q]); dwx = A::sub(vb.w[q], va.w[q]);
                    duz = diff_hi<A>(va.u, q, nu); dwz = diff_hi<A>(va.w, q, nw);
                } else {
                    dux = A::sub(va.u[q], vb.u[q]); dwx = A::sub(va.w[q], vb.w[q]);
                    duz = diff_lo<A>(va.u, q, nu); dwz = diff_lo<A>(va.w, q, nw);
                }
                const f2 u_x = A::mul(dux, idx2, nz2), u_z = A::mul(duz, idz2, nz2);  // fm:369-370, bm:366-367
                const f2 w_x = A::mul(dwx, idx2, nz2), w_z = A::mul(dwz, idz2, nz2);  // fm:371-372, bm:368-369
                const f2 ld = A::mul(m.lam[q], A::add(u_x, w_z), nz2), mu2 = A::add(m.mu[q], m.mu[q]);
                f2 dxx = A::mul(sdt2, A::add(ld, A::mul(mu2, u_x, nz2)), nz2);
                f2 dzz = A::mul(sdt2, A::add(ld, A::mul(mu2, w_z, nz2)), nz2);
                f2 dxz = A::mul(A::mul(sdt2, m.mxz[q], nz2), A::add(u_z, w_x), nz2);
                if constexpr (FAST) {
                    os.xx[q] = A::add(base.xx[q], dxx);
                    os.zz[q] = A::add(base.zz[q], dzz);
                    os.xz[q] = A::add(base.xz[q], dxz);
                    ov.u[q] = va.u[q];
                    ov.w[q] = va.w[q];
                } else {
                    dxx = clip(dxx, q, rm); dzz = clip(dzz, q, rm); dxz = clip(dxz, q, rm);
                    os.xx[q] = A::mul(c, A::add(base.xx[q], dxx), nz2);
                    os.zz[q] = A::mul(A::mul(c, A::add(base.zz[q], dzz), nz2), m.sm[q], nz2);
                    os.xz[q] = A::mul(A::mul(c, A::add(base.xz[q], dxz), nz2), m.sm[q], nz2);
                    ov.u[q] = A::mul(c, va.u[q], nz2);
                    ov.w[q] = A::mul(c, va.w[q], nz2);
                }
            }
            if constexpr (SH) {
                f2 dvx, dvz;
                if constexpr (DIR == 0) { dvx = A::sub(vb.v[q], va.v[q]); dvz = diff_hi<A>(va.v, q, nv); }
                else { dvx = A::sub(va.v[q], vb.v[q]); dvz = diff_lo<A>(va.v, q, nv); }
                const f2 v_x = A::mul(dvx, idx2, nz2), v_z = A::mul(dvz, idz2, nz2);  // fm:381-382, bm:377-378
                f2 dyx = A::mul(A::mul(sdt2, m.myx[q], nz2), v_x, nz2);
                f2 dyz = A::mul(A::mul(sdt2, m.myz[q], nz2), v_z, nz2);
                if constexpr (FAST) {
                    os.yx[q] = A::add(base.yx[q], dyx);
                    os.yz[q] = A::add(base.yz[q], dyz);
                    ov.v[q] = va.v[q];
                } else {
                    dyx = clip(dyx, q, rm); dyz = clip(dyz, q, rm);
                    os.yx[q] = A::mul(c, A::add(base.yx[q], dyx), nz2);
                    os.yz[q] = A::mul(A::mul(c, A::add(base.yz[q], dyz), nz2), m.sm[q], nz2);
                    ov.v[q] = A::mul(c, va.v[q], nz2);
                }
            }
        }
    };
    auto stress_update = [&](int r, const Vel &va, const Vel &vb, const Sig &base, const Mat &m, Sig &os,
                             Vel &ov) {
        float nu = 0.f, nw = 0.f, nv = 0.f;
        if constexpr (DIR == 0) {
            if constexpr (PSV) { nu = __shfl_down_sync(FULL, f2_lo(va.u[0]), 1); nw = __shfl_down_sync(FULL, f2_lo(va.w[0]), 1); }
            if constexpr (SH) nv = __shfl_down_sync(FULL, f2_lo(va.v[0]), 1);
        } else {
            if constexpr (PSV) { nu = __shfl_up_sync(FULL, f2_hi(va.u[NP - 1]), 1); nw = __shfl_up_sync(FULL, f2_hi(va.w[NP - 1]), 1); }
            if constexpr (SH) nv = __shfl_up_sync(FULL, f2_hi(va.v[NP - 1]), 1);
        }
        if (all_in(r) && all_far(r) && p.surface == nullptr)
            stress_cells(std::true_type{}, r, va, vb, base, m, os, ov, nu, nw, nv);
        else
            stress_cells(std::false_type{}, r, va, vb, base, m, os, ov, nu, nw, nv);
    };

    // Per-step outputs of an absorbed velocity row r (owner lanes, r in
    // [ia, ib)): forward receivers at time t and snapshot slot k, backward
    // Kahan imaging against snapshot slot k.
    auto epilogue = [&](int r, int t, int k, const Vel &v) {
        if constexpr (DIR == 0) {
            const int e0 = no_rec ? 0 : ldg_chk(p.rec_ptr + sh.rec_row0 + r);
            const int e1 = no_rec ? 0 : ldg_chk(p.rec_ptr + sh.rec_row0 + r + 1);
            for (int e = e0; e < e1; ++e) {
                const int2 en = ldg_chk(p.rec_ent + e);
                const int q = en.x - c0;
                if (q < 0 || q >= VEC) continue;
                const size_t ti = (size_t)t * p.nrec_total + en.y;
                auto pick = [&](const f2 (&x)[NP]) {
                    const f2 t = NP == 1 || q < 2 ? x[0] : x[NP - 1];
                    return q & 1 ? f2_hi(t) : f2_lo(t);
                };
                if constexpr (PSV) { st_chk(p.seis[0] + ti, pick(v.u)); st_chk(p.seis[2] + ti, pick(v.w)); }
                if constexpr (SH) st_chk(p.seis[1] + ti, pick(v.v));
            }
            if (k >= 0) {
                const long long o = ((long long)p.nsnap * sh.row_off + (long long)k * nx + r) * P + c0 + COL_OFF;
                if constexpr (PSV) { stp<NP>(p.snap[0] + o, v.u); stp<NP>(p.snap[2] + o, v.w); }
                if constexpr (SH) stp<NP>(p.snap[1] + o, v.v);
            }
        } else {
            if (k >= 0) {
                const long long o = ((long long)p.nsnap * sh.row_off + (long long)k * nx + r) * P + c0 + COL_OFF;
                const long long io = (sh.row_off + r) * (long long)P + c0 + COL_OFF;
                auto image = [&](int c, const f2 (&ov2)[NP]) {
                    float s[VEC], sum[VEC], cmp[VEC], ov[VEC];
                    unpack<NP>(ov, ov2);
                    ldv<VEC>(s, p.snap[c] + o);
                    ldv_coherent<VEC>(sum, p.img[c] + io);
                    ldv_coherent<VEC>(cmp, p.imgc[c] + io);
#pragma unroll
                    for (int q = 0; q < VEC; ++q) kahan_add(sum[q], cmp[q], __fmul_rn(s[q], ov[q]));
                    stv<VEC>(p.img[c] + io, sum);
                    stv<VEC>(p.imgc[c] + io, cmp);
                };
                if constexpr (PSV) { image(0, v.u); image(2, v.w); }
                if constexpr (SH) image(1, v.v);
            }
        }
    };

    int code = 0;
    auto check_row = [&](const Vel &v) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            auto bad = [&](f2 x, int c) { code = max(code, max(bad_code(f2_lo(x), c), bad_code(f2_hi(x), c))); };
            if constexpr (PSV) { bad(v.u[q], p.code_base); bad(v.w[q], p.code_base + 2); }
            if constexpr (SH) bad(v.v[q], p.code_base + 1);
        }
    };
    // step A's stress and absorbed velocity of row r (STOREA)
    auto store_a = [&](int r, const Sig &os, const Vel &ov) {
        const long long so = soff + (long long)(r + 1) * P;
        if constexpr (PSV) {
            stp<NP>(p.souta[F_SXX] + so, os.xx);
            stp<NP>(p.souta[F_SZZ] + so, os.zz);
            stp<NP>(p.souta[F_SXZ] + so, os.xz);
            stp<NP>(p.souta[F_U] + so, ov.u);
            stp<NP>(p.souta[F_W] + so, ov.w);
        }
        if constexpr (SH) {
            stp<NP>(p.souta[F_SYX] + so, os.yx);
            stp<NP>(p.souta[F_SYZ] + so, os.yz);
            stp<NP>(p.souta[F_V] + so, ov.v);
        }
    };
    (void)store_a;
    // step B's stress and absorbed velocity of row r: store, outputs, check
    auto finish_b = [&](int r, const Sig &os, const Vel &ov) {
        if constexpr (CKPT) {
            float u[VEC], w[VEC], xx[VEC], zz[VEC], xz[VEC];
            unpack<NP>(u, ov.u); unpack<NP>(w, ov.w);
            unpack<NP>(xx, os.xx); unpack<NP>(zz, os.zz); unpack<NP>(xz, os.xz);
            ckpt_pack_row<VEC>(p.ck, soff + (long long)(r + 1) * P, ck_blk0 + (long long)(r + 1) * p.ck.nblk, lane,
                               owner, u, w, xx, zz, xz);
        }
        if (!owner) return;
        const long long so = soff + (long long)(r + 1) * P;
        if constexpr (PSV) {
            stp<NP>(p.sout[F_SXX] + so, os.xx);
            stp<NP>(p.sout[F_SZZ] + so, os.zz);
            stp<NP>(p.sout[F_SXZ] + so, os.xz);
            stp<NP>(p.sout[F_U] + so, ov.u);
            stp<NP>(p.sout[F_W] + so, ov.w);
        }
        if constexpr (SH) {
            stp<NP>(p.sout[F_SYX] + so, os.yx);
            stp<NP>(p.sout[F_SYZ] + so, os.yz);
            stp<NP>(p.sout[F_V] + so, ov.v);
        }
        epilogue(r, p.it2, p.snap_k2, ov);
        if (p.check) check_row(ov);
    };

    const int tA = p.it, tB = p.it2;
    if constexpr (RING) {
        // rolling rows as in the register version below, minus 1/rho and the
        // material, which come from the ring at the point of use
        Sig so_p, so_c, sa_p, sa_c, s_out;
        Vel va_p, va_c, vb_p, vb_c, vo, vabs_c, vabs_p, v_out;
        [[maybe_unused]] int s0 = 0, s1 = 1, s2 = 2;  // state ring slots of rows k, k+1, k+2
        [[maybe_unused]] Sig n_so;
        [[maybe_unused]] Vel n_vo;
        zero_sig(sa_p); zero_sig(sa_c);
        zero_vel(va_p); zero_vel(vb_p); zero_vel(vabs_c); zero_vel(vabs_p);
        load_sig(ia - 2, so_p);
        if constexpr (DIR == 0) {
            // iteration k: A velocity k, A stress k-1, B velocity k-1, B stress k-2;
            // ring rows read: k (1/rho), k-1 (1/rho, material), k-2 (material);
            // issued: row k+1 into the slot of row k-3
            // SR: copy groups in order: material k, state k+1, material k+1, state k+2
            if constexpr (!SR) { load_sig(ia - 1, n_so); load_vel(ia - 1, n_vo); }
            ring_issue(ia - 2);
            if constexpr (SR) state_issue(0, ia - 1);
            ring_issue(ia - 1);
            if constexpr (SR) state_issue(1, ia);
            for (int k = ia - 1; k <= ib + 1; ++k) {
                if constexpr (!SR) {
                    cp_sig(so_c, n_so);
                    cp_vel(vo, n_vo);
                    if (k <= ib) {
                        load_sig(k + 1, n_so);
                        load_vel(k + 1, n_vo);
                    }
                }
                ring_issue(k + 1);
                if constexpr (SR) {
                    state_issue(s2, k + 2);
                    cp_async_wait<3>();  // material and state up to row k have landed
                    rd_state(s0, so_c, vo);
                    { const int t = s0; s0 = s1; s1 = s2; s2 = t; }
                } else {
                    cp_async_wait<1>();  // every material row up to k has landed
                }
                {
                    Vel ir;
                    ring_ir(k, ir);
                    vel_update(k, tA, so_c, so_p, vo, ir, va_c);
                }
                if (k >= ia) {
                    Mat m;
                    ring_mat(k - 1, m);
                    stress_update(k - 1, va_p, va_c, so_p, m, sa_c, vabs_c);
                    if (owner && k - 1 >= ia && k - 1 < ib) {
                        epilogue(k - 1, tA, p.snap_k, vabs_c);
                        if constexpr (STOREA) store_a(k - 1, sa_c, vabs_c);
                    }
                }
                if (k >= ia + 1) {
                    Vel ir;
                    ring_ir(k - 1, ir);
                    vel_update(k - 1, tB, sa_c, sa_p, vabs_c, ir, vb_c);
                }
                if (k >= ia + 2) {
                    Mat m;
                    ring_mat(k - 2, m);
                    stress_update(k - 2, vb_p, vb_c, sa_p, m, s_out, v_out);
                    finish_b(k - 2, s_out, v_out);
                }
                cp_sig(so_p, so_c);
                cp_vel(va_p, va_c);
                cp_sig(sa_p, sa_c);
                cp_vel(vb_p, vb_c);
            }
        } else {
            // iteration k: A velocity k-1, A stress k-1, B velocity k-2, B stress k-2;
            // ring rows read: k-1, k-2; issued: row k into the slot of row k-4
            load_sig(ia - 1, n_so);
            load_vel(ia - 2, n_vo);
            ring_issue(ia - 2);
            for (int k = ia - 1; k <= ib + 1; ++k) {
                cp_sig(so_c, n_so);   // row k
                cp_vel(vo, n_vo);     // row k-1
                if (k <= ib) {
                    load_sig(k + 1, n_so);
                    load_vel(k, n_vo);
                }
                ring_issue(k);
                cp_async_wait<1>();  // every row up to k-1 has landed
                {
                    Vel ir;
                    ring_ir(k - 1, ir);
                    vel_update(k - 1, tA, so_c, so_p, vo, ir, va_c);
                }
                if (k >= ia) {
                    Mat m;
                    ring_mat(k - 1, m);
                    stress_update(k - 1, va_c, va_p, so_p, m, sa_c, vabs_c);
                    if (owner && k - 1 >= ia && k - 1 < ib) epilogue(k - 1, tA, p.snap_k, vabs_c);
                }
                if (k >= ia + 1) {
                    Vel ir;
                    ring_ir(k - 2, ir);
                    vel_update(k - 2, tB, sa_c, sa_p, vabs_p, ir, vb_c);
                }
                if (k >= ia + 2) {
                    Mat m;
                    ring_mat(k - 2, m);
                    stress_update(k - 2, vb_c, vb_p, sa_p, m, s_out, v_out);
                    finish_b(k - 2, s_out, v_out);
                }
                cp_sig(so_p, so_c);
                cp_vel(va_p, va_c);
                cp_sig(sa_p, sa_c);
                cp_vel(vabs_p, vabs_c);
                cp_vel(vb_p, vb_c);
            }
        }
        cp_async_wait<0>();  // no copy outlives the kernel
    } else {
        // rolling rows (see the header comment for which row each holds)
        Sig so_p, so_c, sa_p, sa_c, s_out, n_so;
        Vel va_p, va_c, vb_p, vb_c, vo, ir_p, ir_c, vabs_c, v_out, n_vo, n_ir;
        Mat m_p, m_c, n_m;
        zero_sig(sa_p); zero_sig(sa_c);
        zero_vel(va_p); zero_vel(vb_p); zero_vel(vabs_c);
        load_sig(ia - 2, so_p);

        if constexpr (DIR == 0) {
            // iteration k: A velocity k, A stress k-1, B velocity k-1, B stress k-2
            // prefetched per iteration: old stress, old velocity, 1/rho of row k+1; material of row k
            load_sig(ia - 1, n_so);
            load_vel(ia - 1, n_vo);
            load_ir(ia - 1, n_ir);
            load_mat(ia - 2, n_m);
            for (int k = ia - 1; k <= ib + 1; ++k) {
                cp_sig(so_c, n_so);
                cp_vel(vo, n_vo);
                cp_vel(ir_c, n_ir);
                cp_mat(m_c, n_m);  // row k-1
                if (k <= ib) {
                    load_sig(k + 1, n_so);
                    load_vel(k + 1, n_vo);
                    load_ir(k + 1, n_ir);
                    load_mat(k, n_m);
                }
                vel_update(k, tA, so_c, so_p, vo, ir_c, va_c);
                if (k >= ia) {
                    stress_update(k - 1, va_p, va_c, so_p, m_c, sa_c, vabs_c);
                    if (owner && k - 1 >= ia && k - 1 < ib) {
                        epilogue(k - 1, tA, p.snap_k, vabs_c);
                        if constexpr (STOREA) store_a(k - 1, sa_c, vabs_c);
                    }
                }
                if (k >= ia + 1) vel_update(k - 1, tB, sa_c, sa_p, vabs_c, ir_p, vb_c);
                if (k >= ia + 2) {
                    stress_update(k - 2, vb_p, vb_c, sa_p, m_p, s_out, v_out);
                    finish_b(k - 2, s_out, v_out);
                }
                cp_sig(so_p, so_c);
                cp_vel(va_p, va_c);
                cp_sig(sa_p, sa_c);
                cp_vel(vb_p, vb_c);
                cp_vel(ir_p, ir_c);
                cp_mat(m_p, m_c);
            }
        } else {
            // iteration k: A velocity k-1, A stress k-1, B velocity k-2, B stress k-2
            // prefetched per iteration: old stress of row k+1; old velocity, 1/rho, material of row k
            Vel vabs_p;
            zero_vel(vabs_p);
            load_sig(ia - 1, n_so);
            load_vel(ia - 2, n_vo);
            load_ir(ia - 2, n_ir);
            load_mat(ia - 2, n_m);
            for (int k = ia - 1; k <= ib + 1; ++k) {
                cp_sig(so_c, n_so);   // row k
                cp_vel(vo, n_vo);     // row k-1
                cp_vel(ir_c, n_ir);   // row k-1
                cp_mat(m_c, n_m);     // row k-1
                if (k <= ib) {
                    load_sig(k + 1, n_so);
                    load_vel(k, n_vo);
                    load_ir(k, n_ir);
                    load_mat(k, n_m);
                }
                vel_update(k - 1, tA, so_c, so_p, vo, ir_c, va_c);
                if (k >= ia) {
                    stress_update(k - 1, va_c, va_p, so_p, m_c, sa_c, vabs_c);
                    if (owner && k - 1 >= ia && k - 1 < ib) epilogue(k - 1, tA, p.snap_k, vabs_c);
                }
                if (k >= ia + 1) vel_update(k - 2, tB, sa_c, sa_p, vabs_p, ir_p, vb_c);
                if (k >= ia + 2) {
                    stress_update(k - 2, vb_c, vb_p, sa_p, m_p, s_out, v_out);
                    finish_b(k - 2, s_out, v_out);
                }
                cp_sig(so_p, so_c);
                cp_vel(va_p, va_c);
                cp_sig(sa_p, sa_c);
                cp_vel(vabs_p, vabs_c);
                cp_vel(vb_p, vb_c);
                cp_vel(ir_p, ir_c);
                cp_mat(m_p, m_c);
            }
        }
    }
    if (p.check) {
        code = __reduce_max_sync(FULL, code);
        if (lane == 0 && code > 0) report_failure(p, wk.x, code);
    }
}

}  // namespace rtm

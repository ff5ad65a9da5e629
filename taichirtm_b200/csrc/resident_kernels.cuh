// Resident propagation: a whole time loop in one cooperative launch, the
// wavefield in registers and the material in shared memory.
//
// A shot's window is cut into tiles, one CTA each.  A CTA's warps are stacked
// over the rows: a warp holds R rows x 64 columns, lane L the column pair
// (2L, 2L+1) of every row, so every neighbour of a stencil is in the lane's own
// registers (rows), one shuffle away (columns) or in a row published by the
// warp above or below through shared memory (two barriers per time step).  The
// tile's outer ring of H rows and columns is halo: it is advanced redundantly,
// loses one ring of validity per step and is refreshed from the neighbouring
// tiles every H steps.  For that exchange each CTA writes the H-deep frame of
// its own cells to its outbox in global memory (L2) as 16-byte packets, three
// values and a tag, the number of the exchange; the neighbours poll for the
// packets themselves.  A packet is read and written by single 128-bit accesses,
// so a fitting tag vouches for its values: no fence, no flag (a release fence
// after the frame took 3,600 cycles here, a packet about 2,000 from register to
// register).  Two outboxes alternate: a CTA writes exchange e+2 only after it
// has read all neighbours' packets e+1, which they send after reading e.
// Nothing else of the wavefield or the material touches memory between the
// first and last step.
//
// The arithmetic of every cell is step_kernel's, operation by operation (two
// columns per packed instruction, see f2_mul), so results are bit-identical.
//
// The waits are bounded: after RES_SPIN_LIMIT polls a CTA raises *err and
// leaves, which makes every other CTA leave too (the host returns an error).
// The launch is cooperative, so all CTAs of a launch are resident.
#pragma once
#include <cuda_runtime.h>
#include <limits.h>

#include "f32x2.cuh"
#include "step_kernels.cuh"

namespace rtm {

constexpr int RES_COLS = 64;             // tile columns: 32 lanes x 2
constexpr int RES_HALO = 4;              // H: halo rows / columns, steps per exchange
constexpr int RES_SPIN_LIMIT = 1 << 22;  // polls of one wait, each an L2 round trip: seconds

struct ResParams {
    // geometry, material, source / receiver tables, outputs: as StepParams
    int nz, pitch, nt, fw;
    float src_factor;
    f2 idx2, idz2, dt2, sdt2, nz2;  // packed 1/dx, 1/dz, dt, +-dt (- backward), -0.0
    const float *sponge;
    const ShotDev *shots;
    const float *mat[NMAT];
    const float *surface;
    const int *src_ptr;
    const int2 *src_ent;
    const float *wav[3];
    const int *rec_ptr;
    const int2 *rec_ent;
    int nrec_total;
    float *seis[3];
    const float *obs[3];
    float *snap[3];
    int nsnap;                 // snapshot slots per shot in the buffers
    float *img[3], *imgc[3];
    bool img_chip;             // backward: images kept in shared memory
    int *flags, *fail_seq;     // per shot: status, step + 1 of the first failed check
    int code_base;
    // loop: steps it0 .. it1-1; the time of step it is it (forward) or nt-1-it (backward)
    int it0, it1, check_interval;
    int isnap, snap_base, snap_lo, snap_hi;  // time t = m * isnap, m in [snap_lo, snap_hi]: slot m - snap_base
    bool segment;              // part of a loop: shots stopped earlier are left alone
    // state: loaded from load[] (null: zero), owned cells stored to store[] at the end (null: not)
    const float *load[NFIELD];
    float *store[NFIELD];
    // forward, keep_every > 0: the state after every keep_every'th step of the launch
    // before nt is stored instead, the first to store[], the next keep floats on, ...
    int keep_every;
    long long keep;
    // tiles
    const int4 *tiles;         // (shot, first owned row, first owned column, wave type); a shot's tiles row by row
    const int4 *shot_tiles;    // per shot, P-SV and SH: (tiles of the shot, tile rows, tile columns, unused)
    int tile0;                 // first tile of this launch
    uint4 *outbox;             // per CTA of the launch: box_stride packets, two outboxes of ResSmem::BOX
    int box_stride;
    unsigned tag0;             // exchange b of this launch is tagged tag0 + b
    unsigned long long *arrive;  // per shot, odd and even checks: tiles that made it | tiles that failed it << 32
    int *err;                  // a wait ran out: in this call, since the host last reported it
    int max_inj, max_rec;      // point entries a tile may hold (host-checked)
#ifdef RTM_BOUNDS_CHECK
    int polls0;                // where a wait starts to count its polls
#endif
};

// Shared memory of one CTA, as byte offsets: per-cell material of NW * R rows x
// 32 lanes, the rows that warps publish to each other, the row descriptors of
// the point entries, then what depends on the plan (entries, staged values,
// surface mask).
template <int MODE, int R, int NW>
struct ResSmem {
    static_assert(MODE == 1 || MODE == 2, "a tile is P-SV or SH");
    static constexpr int CELLS = NW * R * 32, ROWS = NW * R;
    static constexpr int NC = MODE == 1 ? 2 : 1;                     // velocity components
    static constexpr int IR = 0;                                     // P-SV (1/rho_u, 1/rho_w), 16 B
    static constexpr int LM = IR + (MODE == 1 ? CELLS * 16 : 0);    // (lam, 2 mu)
    static constexpr int MY = LM + (MODE == 1 ? CELLS * 16 : 0);    // SH (sdt myx, sdt myz)
    static constexpr int XZ = MY + (MODE == 2 ? CELLS * 16 : 0);    // sdt mxz, 8 B
    static constexpr int IV = XZ + (MODE == 1 ? CELLS * 8 : 0);     // 1/rho
    static constexpr int C = IV + (MODE == 2 ? CELLS * 8 : 0);      // sponge
    static constexpr int VEL = C + CELLS * 8;                        // [comp][warp + 1][lane]
    static constexpr int SIG = VEL + (NW + 2) * 32 * 8 * NC;         // xx, xz / yx
    // exchange: owned rows and lanes, floats and packets of a lane's pair, halo
    // packets of a tile (their values are staged over VEL and SIG, idle then)
    static constexpr int ORW = ROWS - 2 * RES_HALO, OLN = 32 - RES_HALO;
    static constexpr int NF = MODE == 1 ? 10 : 6, NP = (NF + 2) / 3;
    static constexpr int NPAIR = MODE == 1 ? 3 : 2;                  // packets that carry a whole pair
    static constexpr int BOX = ORW * OLN * NP;
    static constexpr int STAGE = (2 * RES_HALO * 32 + ORW * RES_HALO) * NF * 4, ROWBUF = 2 * (NW + 2) * 32 * 8 * NC;
    static constexpr int INFO = VEL + ((STAGE > ROWBUF ? STAGE : ROWBUF) + 15) / 16 * 16;  // ResInfo
    static constexpr int PT = INFO + 80;                             // point table: 16 bits per (row, lane)
    static constexpr int IP = PT + ROWS * 32 * 2;                    // row offsets of the entries
    static constexpr int RP = IP + (ROWS + 2) * 4;
    static constexpr int VAR = (RP + (ROWS + 2) * 4 + 15) / 16 * 16;
    static size_t bytes(bool surface, int max_inj, int max_rec) {
        return VAR + (size_t)max_inj * 8 + (size_t)max_rec * 8 + (size_t)RES_HALO * NC * max_inj * 4 + (surface ? CELLS * 8 : 0);
    }
    // images on the chip: sum, compensation and the next snapshot of each component
    static size_t image_bytes() { return (size_t)CELLS * NC * 3 * 8; }
};

// The point table says for each pair of cells which receiver entry it holds
// (index << 1 | column), RES_NONE, or RES_MANY: more than one (walk the row's).
constexpr unsigned short RES_NONE = 0xffff, RES_MANY = 0xfffe;
constexpr int RES_MAX_POINTS = 0x7ff0;  // receiver entries a tile may hold

// What the exchange and the output rows need of a tile, kept in shared memory
// so that it does not occupy registers between them.
struct ResInfo {
    long long state_off, snap_off, img_off;  // of a shot's state; of tile cell (0, 0) in snapshot slot 0 and in the images
    int slot;                  // floats of a snapshot slot
    int nx, shot, row0, col0;  // first owned row and column
    int nti, ntj;              // the shot's tile rows and columns
    int tiles;                 // tiles of the shot, of both wave types
    int leave;                 // 1: a wait ran out, 2: the shot failed its check
    int bad;                   // this tile failed its check
};
static_assert(sizeof(ResInfo) <= 80, "");

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// One packet by a single (single-copy atomic) 128-bit access.
struct Packet {
    f2 pair, rest;  // rest: the third value, the tag
    __device__ __forceinline__ unsigned tag() const { return (unsigned)(rest >> 32); }
};
__device__ __forceinline__ void ld_packet(Packet &v, const uint4 *p) {
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(v.pair), "=l"(v.rest) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_packet(uint4 *p, f2 pair, float z, unsigned tag) {
    const f2 b = f2_pack(z, __uint_as_float(tag));
    asm volatile("{ .reg .b128 t; mov.b128 t, {%0, %1}; st.relaxed.gpu.global.b128 [%2], t; }" ::"l"(pair), "l"(b), "l"(p) : "memory");
}
// x = *p (shared memory) where the predicate holds: without a branch, so that
// the loads of all rows are in flight together
__device__ __forceinline__ void lds_if(f2 &x, unsigned addr, bool pred) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.shared.b64 %0, [%1]; }" : "+l"(x) : "r"(addr), "r"((unsigned)pred) : "memory");
}

// *p = x where the predicate holds, without a branch
__device__ __forceinline__ void st_if(float *p, float x, bool pred) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q st.global.f32 [%0], %1; }" ::"l"(p), "f"(x), "r"((unsigned)pred) : "memory");
}

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// CTAs per SM that the register budget is cut for: the wavefield takes 2 R
// registers per field (5 P-SV, 3 SH), the arithmetic of a row about 40 more.  At
// these budgets most kernels spill some (the table of layouts in rtm_api.cu has
// the bytes).
template <int MODE, int R, int NW>
constexpr int res_ctas() {
    constexpr int state = 2 * R * (MODE == 1 ? 5 : 3);
    return (state <= 30 ? 32 : state <= 40 ? 24 : 16) / NW;
}

extern __shared__ __align__(16) unsigned char res_smem_raw[];

template <int DIR, int MODE, int R, int NW>
__device__ __forceinline__ void resident_body(const ResParams &p) {
    using L = ResSmem<MODE, R, NW>;
    constexpr bool PSV = MODE == 1, SH = MODE == 2;
    constexpr int NC = L::NC;
    constexpr int RT = L::ROWS;
    const int lane = threadIdx.x & 31;
    const int warp = __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0);  // known to be the same on every lane

    unsigned char *const sm0 = res_smem_raw;
    volatile ResInfo *const info = reinterpret_cast<volatile ResInfo *>(sm0 + L::INFO);
    unsigned short *const s_pt = reinterpret_cast<unsigned short *>(sm0 + L::PT);
    int *const s_ip = reinterpret_cast<int *>(sm0 + L::IP), *const s_rp = reinterpret_cast<int *>(sm0 + L::RP);
    int2 *const s_inj = reinterpret_cast<int2 *>(sm0 + L::VAR);  // (tile row << 8 | column, index)
    auto s_rec = [&]() { return s_inj + p.max_inj; };
    auto s_val = [&]() { return reinterpret_cast<float *>(s_inj + p.max_inj + p.max_rec); };  // [step][comp][entry]
    auto s_sm = [&]() { return reinterpret_cast<f2 *>(s_val() + (size_t)RES_HALO * NC * p.max_inj); };
    // this lane's cell of row 0; row r is 32 cells on
    const int cell0 = warp * (R * 32) + lane;
    unsigned char *const c16 = sm0 + cell0 * 16, *const c8 = sm0 + cell0 * 8;
    // image rows (img_chip): [component][sum, compensation, snapshot][cell]
    auto s_img = [&](int comp, int what, int r) -> f2 & {
        f2 *b = s_sm() + (p.surface ? L::CELLS : 0);
        return b[(size_t)(comp * 3 + what) * L::CELLS + cell0 + 32 * r];
    };
    auto at16 = [&](int off, int r) { return *reinterpret_cast<const ulonglong2 *>(c16 + off + r * 512); };
    auto at8 = [&](int off, int r) { return *reinterpret_cast<const f2 *>(c8 + off + r * 256); };
    // this warp's published row of component comp; the warps above and below: -256, +256 bytes
    unsigned char *const wrow = sm0 + (warp + 1) * 256 + lane * 8;
    auto pub = [&](int off, int comp, int d) -> f2 & {
        return *reinterpret_cast<f2 *>(wrow + off + comp * ((NW + 2) * 256) + d * 256);
    };
    const f2 nz2 = p.nz2;

    // ---- set-up: material, sponge, masks and point entries of the tile
    unsigned cm0, cm1;     // column masks: all ones for an interior column (1 <= j <= nz-2)
    unsigned row_bits = 0;  // bit r: row r is interior (1 <= i <= nx-2)
    int kind;              // per warp: 0 interior, no sponge; 1 sponge; 2 edge cells; 3 surface mask
    bool sources;           // forward: this warp's rows hold sources
    int points = 0;         // receivers in this warp's rows: 0 none, 1 by the table, 2 by the lists
    {
        const int4 tl = p.tiles[p.tile0 + blockIdx.x];
        const int4 st = p.shot_tiles[2 * tl.x + (PSV ? 0 : 1)];
        const ShotDev sh = p.shots[tl.x];
        const int nx = sh.nx, nz = p.nz, P = p.pitch;
        constexpr int H = RES_HALO;
        const int row0 = tl.y - H + warp * R, col = tl.z - H + 2 * lane;
        // a failure of this launch is later than it0, so all tiles agree
        if (p.segment && ld_acquire(p.fail_seq + tl.x) <= p.it0) return;
        if (threadIdx.x == 0) {
            info->state_off = sh.state_off;
            const long long at = (long long)(tl.y - H) * P + (tl.z - H) + COL_OFF;
            info->snap_off = (long long)p.nsnap * sh.row_off * P + at;
            info->img_off = sh.row_off * P + at;
            info->slot = nx * P;
            info->nx = nx;
            info->shot = tl.x;
            info->row0 = tl.y;
            info->col0 = tl.z;
            info->nti = st.y;
            info->ntj = st.z;
            info->tiles = st.x;
            info->leave = info->bad = 0;
        }
        cm0 = (unsigned)(col - 1) < (unsigned)(nz - 2) ? ~0u : 0u;
        cm1 = (unsigned)col < (unsigned)(nz - 2) ? ~0u : 0u;
        // kept as bit masks: a known all-or-nothing value would turn the ANDs of
        // clip() back into compares and selects
        asm volatile("" : "+r"(cm0), "+r"(cm1));
        bool edge = false, absorb = false, masked = false;
        StepParams spg;  // what sponge_coef reads
        spg.fw = p.fw;
        spg.nz = nz;
        spg.sponge = p.sponge;
        const float sdt = f2_lo(p.sdt2);
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            const int i = row0 + r;
            float ir[2][2] = {}, lm[2][2] = {}, xz[2] = {}, my[2][2] = {}, iv[2] = {}, c[2] = {1.f, 1.f}, sm[2] = {1.f, 1.f};
            if ((unsigned)(i - 1) < (unsigned)(nx - 2)) row_bits |= 1u << r;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = col + q;
                edge = edge || !interior(i, j, nx, nz);
                if ((unsigned)i >= (unsigned)nx || (unsigned)j >= (unsigned)nz) continue;
                const long long mo = (long long)(sh.x0 + i + 1) * P + j + COL_OFF;
                if constexpr (PSV) {
                    ir[0][q] = ldg_chk(p.mat[M_IRU] + mo);
                    ir[1][q] = ldg_chk(p.mat[M_IRW] + mo);
                    lm[0][q] = ldg_chk(p.mat[M_LAM] + mo);
                    lm[1][q] = 2.0f * ldg_chk(p.mat[M_MU] + mo);
                    xz[q] = sdt * ldg_chk(p.mat[M_MXZ] + mo);
                }
                if constexpr (SH) {
                    my[0][q] = sdt * ldg_chk(p.mat[M_MYX] + mo);
                    my[1][q] = sdt * ldg_chk(p.mat[M_MYZ] + mo);
                    iv[q] = ldg_chk(p.mat[M_IR] + mo);
                }
                c[q] = sponge_coef(spg, nx, i, j);
                if (p.surface) sm[q] = ldg_chk(p.surface + mo);
                absorb = absorb || c[q] != 1.0f;
                masked = masked || sm[q] != 1.0f;
            }
            auto put16 = [&](int off, float a, float b, float cc, float d) {
                *reinterpret_cast<float4 *>(c16 + off + r * 512) = make_float4(a, b, cc, d);
            };
            auto put8 = [&](int off, float a, float b) {
                *reinterpret_cast<float2 *>(c8 + off + r * 256) = make_float2(a, b);
            };
            if constexpr (PSV) {
                put16(L::IR, ir[0][0], ir[0][1], ir[1][0], ir[1][1]);
                put16(L::LM, lm[0][0], lm[0][1], lm[1][0], lm[1][1]);
                put8(L::XZ, xz[0], xz[1]);
            }
            if constexpr (SH) {
                put16(L::MY, my[0][0], my[0][1], my[1][0], my[1][1]);
                put8(L::IV, iv[0], iv[1]);
            }
            put8(L::C, c[0], c[1]);
            if (p.surface) s_sm()[cell0 + 32 * r] = f2_pack(sm[0], sm[1]);
        }
        kind = __any_sync(FULL, masked) ? 3 : __any_sync(FULL, edge) ? 2 : __any_sync(FULL, absorb) ? 1 : 0;
        for (int k = threadIdx.x; k < 2 * (NW + 2) * 32 * NC; k += 32 * NW) reinterpret_cast<f2 *>(sm0 + L::VEL)[k] = 0ull;

        // point entries, row by row in table order: injection (forward sources,
        // backward observed data) on every cell of the tile, recording (forward
        // receivers) on owned cells
        const int *inj_ptr = DIR == 0 ? p.src_ptr + sh.src_row0 : p.rec_ptr + sh.rec_row0;
        const int2 *inj_ent = DIR == 0 ? p.src_ent : p.rec_ent;
        auto row_entries = [&](const int *ptr, const int2 *ent, int rr, bool own, int2 *out, int cap) {
            const int i = tl.y - H + rr;
            if ((unsigned)i >= (unsigned)nx || (own && (rr < H || rr >= RT - H))) return 0;
            const int lo = tl.z - (own ? 0 : H), hi = tl.z - H + RES_COLS - (own ? H : 0);
            int n = 0;
            for (int e = ldg_chk(ptr + i), e1 = ldg_chk(ptr + i + 1); e < e1; ++e) {
                const int2 en = ldg_chk(ent + e);
                if (en.x < lo || en.x >= hi) continue;
                if (out && n < cap) out[n] = make_int2(rr << 8 | (en.x - (tl.z - H)), en.y);
                ++n;
            }
            return n;
        };
        for (int rr = threadIdx.x; rr < RT; rr += 32 * NW) {
            s_ip[rr] = row_entries(inj_ptr, inj_ent, rr, false, nullptr, 0);
            if (DIR == 0) s_rp[rr] = p.seis[PSV ? 0 : 1] ? row_entries(p.rec_ptr + sh.rec_row0, p.rec_ent, rr, true, nullptr, 0) : 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int a = 0, b = 0;
            for (int rr = 0; rr < RT; ++rr) {
                const int n = s_ip[rr];
                s_ip[rr] = a;
                a = min(a + n, p.max_inj);
                if (DIR == 0) {
                    const int m = s_rp[rr];
                    s_rp[rr] = b;
                    b = min(b + m, p.max_rec);
                }
            }
            s_ip[RT] = a;
            s_rp[RT] = b;
        }
        __syncthreads();
        for (int rr = threadIdx.x; rr < RT; rr += 32 * NW) {
            const int a = s_ip[rr], n = s_ip[rr + 1] - a;
            row_entries(inj_ptr, inj_ent, rr, false, s_inj + a, n);
            const int b = DIR == 0 ? s_rp[rr] : a, m = DIR == 0 ? s_rp[rr + 1] - b : n;
            const int2 *ent = DIR == 0 ? s_rec() + b : s_inj + a;
            if (DIR == 0 && m) row_entries(p.rec_ptr + sh.rec_row0, p.rec_ent, rr, true, s_rec() + b, m);
            unsigned short *t = s_pt + rr * 32;
            for (int l = 0; l < 32; ++l) t[l] = RES_NONE;
            for (int e = 0; e < m; ++e) {
                const int l = (ent[e].x & 255) >> 1;
                t[l] = t[l] == RES_NONE ? (unsigned short)((b + e) << 1 | (ent[e].x & 1)) : RES_MANY;
            }
        }
        __syncthreads();
        for (int r = 0; r < R; ++r) {
            const unsigned t = s_pt[(warp * R + r) * 32 + lane];
            points = max(points, t == RES_MANY ? 2 : t != RES_NONE ? 1 : 0);
        }
        sources = DIR == 0 && s_ip[(warp + 1) * R] > s_ip[warp * R];
        points = __reduce_max_sync(FULL, points);
    }

    // ---- state
    f2 U[PSV ? R : 1], W[PSV ? R : 1], XX[PSV ? R : 1], ZZ[PSV ? R : 1], XZ[PSV ? R : 1];
    f2 V[SH ? R : 1], YX[SH ? R : 1], YZ[SH ? R : 1];
    auto ld2 = [&](const float *b, long long o) -> f2 {
        if (!RTM_DBG_OK(b + o, 8)) return 0ull;
        return __ldcg(reinterpret_cast<const unsigned long long *>(b + o));
    };
    auto st2 = [&](float *b, long long o, f2 v) {
        if (!RTM_DBG_OK(b + o, 8)) return;
        *reinterpret_cast<unsigned long long *>(b + o) = v;
    };
    // A pair is stored and loaded whole: the second column of the last pair of
    // an odd nz is a padding column, zero in every buffer.
    auto load_row = [&](int r, long long o, const float *const *b) {
        if constexpr (PSV) {
            U[r] = ld2(b[F_U], o); W[r] = ld2(b[F_W], o);
            XX[r] = ld2(b[F_SXX], o); ZZ[r] = ld2(b[F_SZZ], o); XZ[r] = ld2(b[F_SXZ], o);
        }
        if constexpr (SH) { V[r] = ld2(b[F_V], o); YX[r] = ld2(b[F_SYX], o); YZ[r] = ld2(b[F_SYZ], o); }
    };
    auto store_row = [&](int r, long long o, float *const *b) {
        if constexpr (PSV) {
            st2(b[F_U], o, U[r]); st2(b[F_W], o, W[r]);
            st2(b[F_SXX], o, XX[r]); st2(b[F_SZZ], o, ZZ[r]); st2(b[F_SXZ], o, XZ[r]);
        }
        if constexpr (SH) { st2(b[F_V], o, V[r]); st2(b[F_SYX], o, YX[r]); st2(b[F_SYZ], o, YZ[r]); }
    };
    // window row of this warp's row 0, window column of the lane's first column
    auto my_row0 = [&]() { return info->row0 - RES_HALO + warp * R; };
    auto my_col = [&]() { return info->col0 - RES_HALO + 2 * lane; };
    // rows of this warp inside the window and owned: bit masks over r
    auto rows_in = [&](int row0, int nx) {
        unsigned m = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) m |= (unsigned)((unsigned)(row0 + r) < (unsigned)nx) << r;
        return m;
    };
    // bit r: this lane's pair of row r is the tile's own, inside the window
    unsigned own = 0;
    if (lane >= RES_HALO / 2 && lane < 32 - RES_HALO / 2 && my_col() < p.nz) {
        const int row0 = my_row0(), nx = info->nx;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int rr = warp * R + r;
            own |= (unsigned)(rr >= RES_HALO && rr < RT - RES_HALO && row0 + r < nx) << r;
        }
    }
    auto state_at = [&](int row0, int col) { return info->state_off + (long long)(row0 + 1) * p.pitch + (col + COL_OFF); };
    {
        const int row0 = my_row0(), col = my_col(), nx = info->nx;
        const unsigned in = rows_in(row0, nx);
        const long long so = state_at(row0, col);
        const bool have = p.load[PSV ? F_U : F_V] != nullptr && (unsigned)col < (unsigned)p.nz;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (PSV) U[r] = W[r] = XX[r] = ZZ[r] = XZ[r] = 0ull;
            if constexpr (SH) V[r] = YX[r] = YZ[r] = 0ull;
            if (have && (in >> r & 1)) load_row(r, so + (long long)r * p.pitch, p.load);
        }
    }

    // ---- the two half steps
    auto publish_sig = [&]() {
        constexpr int r = DIR == 0 ? R - 1 : 0;
        if constexpr (PSV) { pub(L::SIG, 0, 0) = XX[r]; pub(L::SIG, 1, 0) = XZ[r]; }
        if constexpr (SH) pub(L::SIG, 0, 0) = YX[r];
    };
    auto publish_vel = [&]() {
        constexpr int r = DIR == 0 ? 0 : R - 1;
        if constexpr (PSV) { pub(L::VEL, 0, 0) = U[r]; pub(L::VEL, 1, 0) = W[r]; }
        if constexpr (SH) pub(L::VEL, 0, 0) = V[r];
    };
    // An update of a row with edge cells: cells that are not interior keep their
    // value.  Their increment is cleared bitwise, so not even a NaN gets in.
    auto mask_row = [&](int r) -> unsigned { return (unsigned)((int)(row_bits << (31 - r)) >> 31); };
    auto clip = [&](f2 d, unsigned rm) -> f2 {
        return (f2)((unsigned)(d >> 32) & cm1 & rm) << 32 | ((unsigned)d & cm0 & rm);
    };
    // Velocity update (fm:332-347, bm:333-345): row r reads stress rows r-1, r
    // (forward) or r, r+1 (backward), columns j-1, j or j, j+1.
    auto velocity = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        constexpr int D = DIR == 0 ? -1 : 1;
        [[maybe_unused]] f2 nxx = 0, nxz = 0, nyx = 0;  // the neighbouring warp's stress row
        if constexpr (PSV) { nxx = pub(L::SIG, 0, D); nxz = pub(L::SIG, 1, D); }
        if constexpr (SH) nyx = pub(L::SIG, 0, D);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int r = DIR == 0 ? k : R - 1 - k;
            const bool end = k == 0;
            const int rn = end ? r : r + D;
            unsigned rm = 0;
            if constexpr (EDGE) rm = mask_row(r);
            if constexpr (PSV) {
                const ulonglong2 ir = at16(L::IR, r);
                const f2 xxn = end ? nxx : XX[rn], xzn = end ? nxz : XZ[rn];
                f2 dzz, dxz;
                if constexpr (DIR == 0) {
                    const float zl = __shfl_up_sync(FULL, f2_hi(ZZ[r]), 1), xl = __shfl_up_sync(FULL, f2_hi(XZ[r]), 1);
                    dzz = f2_pack(f2_lo(ZZ[r]) - zl, f2_hi(ZZ[r]) - f2_lo(ZZ[r]));
                    dxz = f2_pack(f2_lo(XZ[r]) - xl, f2_hi(XZ[r]) - f2_lo(XZ[r]));
                } else {
                    const float zr = __shfl_down_sync(FULL, f2_lo(ZZ[r]), 1), xr = __shfl_down_sync(FULL, f2_lo(XZ[r]), 1);
                    dzz = f2_pack(f2_hi(ZZ[r]) - f2_lo(ZZ[r]), zr - f2_hi(ZZ[r]));
                    dxz = f2_pack(f2_hi(XZ[r]) - f2_lo(XZ[r]), xr - f2_hi(XZ[r]));
                }
                const f2 dxx = DIR == 0 ? f2_sub(XX[r], xxn) : f2_sub(xxn, XX[r]);
                const f2 dzx = DIR == 0 ? f2_sub(XZ[r], xzn) : f2_sub(xzn, XZ[r]);
                const f2 sxx_x = f2_mul(dxx, p.idx2, nz2), szz_z = f2_mul(dzz, p.idz2, nz2);
                const f2 sxz_x = f2_mul(dzx, p.idx2, nz2), sxz_z = f2_mul(dxz, p.idz2, nz2);
                f2 du = f2_mul(f2_mul(f2_add(sxx_x, sxz_z), p.dt2, nz2), ir.x, nz2);
                f2 dw = f2_mul(f2_mul(f2_add(sxz_x, szz_z), p.dt2, nz2), ir.y, nz2);
                if constexpr (EDGE) { du = clip(du, rm); dw = clip(dw, rm); }
                U[r] = DIR == 0 ? f2_add(U[r], du) : f2_sub(U[r], du);
                W[r] = DIR == 0 ? f2_add(W[r], dw) : f2_sub(W[r], dw);
            }
            if constexpr (SH) {
                const f2 iv = at8(L::IV, r);
                const f2 yxn = end ? nyx : YX[rn];
                f2 dyz;
                if constexpr (DIR == 0) {
                    const float yl = __shfl_up_sync(FULL, f2_hi(YZ[r]), 1);
                    dyz = f2_pack(f2_lo(YZ[r]) - yl, f2_hi(YZ[r]) - f2_lo(YZ[r]));
                } else {
                    const float yr = __shfl_down_sync(FULL, f2_lo(YZ[r]), 1);
                    dyz = f2_pack(f2_hi(YZ[r]) - f2_lo(YZ[r]), yr - f2_hi(YZ[r]));
                }
                const f2 dyx = DIR == 0 ? f2_sub(YX[r], yxn) : f2_sub(yxn, YX[r]);
                const f2 syx_x = f2_mul(dyx, p.idx2, nz2), syz_z = f2_mul(dyz, p.idz2, nz2);
                f2 dv = f2_mul(f2_mul(f2_add(syx_x, syz_z), p.dt2, nz2), iv, nz2);
                if constexpr (EDGE) dv = clip(dv, rm);
                V[r] = DIR == 0 ? f2_add(V[r], dv) : f2_sub(V[r], dv);
            }
        }
    };
    // Point values by the lists: entry after entry in table order, added to
    // whichever row holds it.  x + -0.0 is x for every x, so rows and lanes
    // without the entry take part and need no branch.
    auto add_at = [&](f2 (&x)[PSV ? R : 1], int row, int c, float a) {
        const f2 v = f2_pack(c == 2 * lane ? a : -0.0f, c == 2 * lane + 1 ? a : -0.0f);
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = f2_add(x[r], r == row ? v : f2_pack(-0.0f, -0.0f));
    };
    auto add_at_v = [&](f2 (&x)[SH ? R : 1], int row, int c, float a) {
        const f2 v = f2_pack(c == 2 * lane ? a : -0.0f, c == 2 * lane + 1 ? a : -0.0f);
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = f2_add(x[r], r == row ? v : f2_pack(-0.0f, -0.0f));
    };
    // sources (fm:421-443) or observed data (bm:452-460) of step s of the block
    auto inject_list = [&](int s) {
        const float *val = s_val() + (size_t)s * NC * p.max_inj;
#pragma unroll 1
        for (int e = s_ip[warp * R]; e < s_ip[(warp + 1) * R]; ++e) {
            const int rc = s_inj[e].x, c = rc & 255, row = (rc >> 8) - warp * R;
            auto scaled = [&](int comp, f2 ir2, bool masked) {
                float a = val[comp * p.max_inj + e];
                if constexpr (DIR == 0) {
                    // 1/rho is +inf at the edge cells of P-SV (fm:306-307)
                    const bool hi = c & 1, in = (row_bits >> row & 1) && (hi ? cm1 : cm0);
                    a = a * p.src_factor * (in || !masked ? (hi ? f2_hi(ir2) : f2_lo(ir2)) : __int_as_float(0x7f800000));
                }
                return a;
            };
            if constexpr (PSV) {
                const ulonglong2 ir = *reinterpret_cast<const ulonglong2 *>(c16 + L::IR + row * 512);
                add_at(U, row, c, scaled(0, ir.x, true));
                add_at(W, row, c, scaled(1, ir.y, true));
            }
            if constexpr (SH) add_at_v(V, row, c, scaled(0, *reinterpret_cast<const f2 *>(c8 + L::IV + row * 256), false));
        }
    };
    // Observed data by the table: one receiver per pair of cells at most.
    auto inject_table = [&](int s) {
        const float *val = s_val() + (size_t)s * NC * p.max_inj;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned t = s_pt[(warp * R + r) * 32 + lane];
            const bool have = t != RES_NONE;
            const int e = have ? t >> 1 : 0;
            auto add = [&](f2 &x, int comp) {
                const float a = val[comp * p.max_inj + e];
                x = f2_add(x, f2_pack(have && !(t & 1) ? a : -0.0f, have && (t & 1) ? a : -0.0f));
            };
            if constexpr (PSV) { add(U[r], 0); add(W[r], 1); }
            if constexpr (SH) add(V[r], 0);
        }
    };
    // Stress update and absorbing (fm:369-419, bm:366-419); KIND as `kind`.
    auto stress = [&](auto kind_tag) {
        constexpr int KIND = decltype(kind_tag)::value;
        constexpr int D = DIR == 0 ? 1 : -1;
        [[maybe_unused]] f2 nu = 0, nw_ = 0, nv = 0;  // the neighbouring warp's velocity row
        if constexpr (PSV) { nu = pub(L::VEL, 0, D); nw_ = pub(L::VEL, 1, D); }
        if constexpr (SH) nv = pub(L::VEL, 0, D);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            // in the order in which row r's raw velocity is last read
            const int r = DIR == 0 ? k : R - 1 - k;
            const bool end = k == R - 1;
            const int rn = end ? r : r + D;
            unsigned rm = 0;
            if constexpr (KIND >= 2) rm = mask_row(r);
            f2 c = 0, sm = 0;
            if constexpr (KIND >= 1) c = at8(L::C, r);
            if constexpr (KIND == 3) sm = s_sm()[cell0 + 32 * r];
            if constexpr (PSV) {
                const ulonglong2 lm = at16(L::LM, r);
                const f2 mx = at8(L::XZ, r);
                const f2 ub = end ? nu : U[rn], wb = end ? nw_ : W[rn];
                f2 duz, dwz;
                if constexpr (DIR == 0) {
                    const float ur = __shfl_down_sync(FULL, f2_lo(U[r]), 1), wr = __shfl_down_sync(FULL, f2_lo(W[r]), 1);
                    duz = f2_pack(f2_hi(U[r]) - f2_lo(U[r]), ur - f2_hi(U[r]));
                    dwz = f2_pack(f2_hi(W[r]) - f2_lo(W[r]), wr - f2_hi(W[r]));
                } else {
                    const float ul = __shfl_up_sync(FULL, f2_hi(U[r]), 1), wl = __shfl_up_sync(FULL, f2_hi(W[r]), 1);
                    duz = f2_pack(f2_lo(U[r]) - ul, f2_hi(U[r]) - f2_lo(U[r]));
                    dwz = f2_pack(f2_lo(W[r]) - wl, f2_hi(W[r]) - f2_lo(W[r]));
                }
                const f2 dux = DIR == 0 ? f2_sub(ub, U[r]) : f2_sub(U[r], ub);
                const f2 dwx = DIR == 0 ? f2_sub(wb, W[r]) : f2_sub(W[r], wb);
                const f2 u_x = f2_mul(dux, p.idx2, nz2), u_z = f2_mul(duz, p.idz2, nz2);
                const f2 w_x = f2_mul(dwx, p.idx2, nz2), w_z = f2_mul(dwz, p.idz2, nz2);
                const f2 ld = f2_mul(lm.x, f2_add(u_x, w_z), nz2);
                f2 dxx = f2_mul(p.sdt2, f2_add(ld, f2_mul(lm.y, u_x, nz2)), nz2);
                f2 dzz = f2_mul(p.sdt2, f2_add(ld, f2_mul(lm.y, w_z, nz2)), nz2);
                f2 dxz = f2_mul(mx, f2_add(u_z, w_x), nz2);
                if constexpr (KIND >= 2) { dxx = clip(dxx, rm); dzz = clip(dzz, rm); dxz = clip(dxz, rm); }
                f2 xx = f2_add(XX[r], dxx), zz = f2_add(ZZ[r], dzz), xz = f2_add(XZ[r], dxz);
                if constexpr (KIND >= 1) {
                    xx = f2_mul(c, xx, nz2);
                    zz = f2_mul(c, zz, nz2);
                    xz = f2_mul(c, xz, nz2);
                    U[r] = f2_mul(c, U[r], nz2);
                    W[r] = f2_mul(c, W[r], nz2);
                }
                if constexpr (KIND == 3) { zz = f2_mul(zz, sm, nz2); xz = f2_mul(xz, sm, nz2); }
                XX[r] = xx; ZZ[r] = zz; XZ[r] = xz;
            }
            if constexpr (SH) {
                const ulonglong2 my = at16(L::MY, r);
                const f2 vb = end ? nv : V[rn];
                f2 dvz;
                if constexpr (DIR == 0) {
                    const float vr = __shfl_down_sync(FULL, f2_lo(V[r]), 1);
                    dvz = f2_pack(f2_hi(V[r]) - f2_lo(V[r]), vr - f2_hi(V[r]));
                } else {
                    const float vl = __shfl_up_sync(FULL, f2_hi(V[r]), 1);
                    dvz = f2_pack(f2_lo(V[r]) - vl, f2_hi(V[r]) - f2_lo(V[r]));
                }
                const f2 dvx = DIR == 0 ? f2_sub(vb, V[r]) : f2_sub(V[r], vb);
                f2 dyx = f2_mul(my.x, f2_mul(dvx, p.idx2, nz2), nz2);
                f2 dyz = f2_mul(my.y, f2_mul(dvz, p.idz2, nz2), nz2);
                if constexpr (KIND >= 2) { dyx = clip(dyx, rm); dyz = clip(dyz, rm); }
                f2 yx = f2_add(YX[r], dyx), yz = f2_add(YZ[r], dyz);
                if constexpr (KIND >= 1) {
                    yx = f2_mul(c, yx, nz2);
                    yz = f2_mul(c, yz, nz2);
                    V[r] = f2_mul(c, V[r], nz2);
                }
                if constexpr (KIND == 3) yz = f2_mul(yz, sm, nz2);
                YX[r] = yx; YZ[r] = yz;
            }
        }
    };
    // Seismograms (fm:445-453), owned cells.
    auto record = [&](int t) {
        const size_t to = (size_t)t * p.nrec_total;
        if (points == 1) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const unsigned tb = s_pt[(warp * R + r) * 32 + lane];
                const bool have = tb != RES_NONE, hi = tb & 1;
                const size_t o = to + s_rec()[have ? tb >> 1 : 0].y;
                auto put = [&](float *q, f2 x) { st_if(q, hi ? f2_hi(x) : f2_lo(x), have && RTM_DBG_OK(q, 4)); };
                if constexpr (PSV) { put(p.seis[0] + o, U[r]); put(p.seis[2] + o, W[r]); }
                if constexpr (SH) put(p.seis[1] + o, V[r]);
            }
        } else {
#pragma unroll 1
            for (int e = s_rp[warp * R]; e < s_rp[(warp + 1) * R]; ++e) {
                const int2 en = s_rec()[e];
                const int row = (en.x >> 8) - warp * R, c = en.x & 255;
                const size_t o = to + en.y;
                auto put = [&](float *q, const f2 *x) {
                    f2 v = x[0];
#pragma unroll
                    for (int r = 1; r < R; ++r) v = r == row ? x[r] : v;
                    st_if(q, c & 1 ? f2_hi(v) : f2_lo(v), (c >> 1) == lane && RTM_DBG_OK(q, 4));
                };
                if constexpr (PSV) { put(p.seis[0] + o, U); put(p.seis[2] + o, W); }
                if constexpr (SH) put(p.seis[1] + o, V);
            }
        }
    };
    // Snapshot slot k (fm:490-497) or its correlation (bm:481-488), owned cells.
    auto snapshot = [&](int k) {
        if (!own) return;
        const long long P = p.pitch;
        const int cell = warp * R * p.pitch + 2 * lane;
        const long long o = info->snap_off + (long long)k * info->slot + cell;
        if constexpr (DIR == 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!(own >> r & 1)) continue;
                if constexpr (PSV) { st2(p.snap[0], o + r * P, U[r]); st2(p.snap[2], o + r * P, W[r]); }
                if constexpr (SH) st2(p.snap[1], o + r * P, V[r]);
            }
        } else {
            // Kahan update.  Two-row tiles load everything before the first store: one
            // L2 round trip instead of one per row and component (the loads cannot be
            // moved over the stores); 301 x 151, an image at every step: 2.70 -> 2.40 ms
            // per 500-step RTM.  Taller ones have no registers for it: the spills
            // cost every step (R 6: 3.0 -> 3.4 us).
            const long long io = info->img_off + cell;
            if (p.img_chip) {
                cp_async_wait<0>();  // this lane's own copies of the snapshot
                auto image = [&](int comp, int r, f2 v) {
                    const f2 sn = s_img(comp, 2, r), im = s_img(comp, 0, r), ic = s_img(comp, 1, r);
                    float s0 = f2_lo(im), c0 = f2_lo(ic), s1 = f2_hi(im), c1 = f2_hi(ic);
                    kahan_add(s0, c0, __fmul_rn(f2_lo(sn), f2_lo(v)));
                    kahan_add(s1, c1, __fmul_rn(f2_hi(sn), f2_hi(v)));
                    s_img(comp, 0, r) = f2_pack(s0, s1);
                    s_img(comp, 1, r) = f2_pack(c0, c1);
                };
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (!(own >> r & 1)) continue;
                    if constexpr (PSV) { image(0, r, U[r]); image(1, r, W[r]); }
                    if constexpr (SH) image(0, r, V[r]);
                }
                return;
            }
            auto update = [&](int c, int r, f2 sn, f2 im, f2 ic, f2 v) {
                float s0 = f2_lo(im), c0 = f2_lo(ic), s1 = f2_hi(im), c1 = f2_hi(ic);
                kahan_add(s0, c0, __fmul_rn(f2_lo(sn), f2_lo(v)));
                kahan_add(s1, c1, __fmul_rn(f2_hi(sn), f2_hi(v)));
                st2(p.img[c], io + r * P, f2_pack(s0, s1));
                st2(p.imgc[c], io + r * P, f2_pack(c0, c1));
            };
            if constexpr (R == 2) {
                constexpr int N = PSV ? 2 : 1;
                f2 sn[R][N], im[R][N], ic[R][N];
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const int c = PSV ? 2 * k : 1;
                        if (!(own >> r & 1)) continue;
                        sn[r][k] = ld2(p.snap[c], o + r * P);
                        im[r][k] = ld2(p.img[c], io + r * P);
                        ic[r][k] = ld2(p.imgc[c], io + r * P);
                    }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (!(own >> r & 1)) continue;
                    if constexpr (PSV) {
                        update(0, r, sn[r][0], im[r][0], ic[r][0], U[r]);
                        update(2, r, sn[r][1], im[r][1], ic[r][1], W[r]);
                    } else {
                        update(1, r, sn[r][0], im[r][0], ic[r][0], V[r]);
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (!(own >> r & 1)) continue;
                    auto image = [&](int c, f2 v) {
                        update(c, r, ld2(p.snap[c], o + r * P), ld2(p.img[c], io + r * P), ld2(p.imgc[c], io + r * P), v);
                    };
                    if constexpr (PSV) { image(0, U[r]); image(2, W[r]); }
                    if constexpr (SH) image(1, V[r]);
                }
            }
        }
    };
    // img_chip: copy snapshot slot k's pairs in (each lane its own, so its own
    // wait is enough), and move the images in or out.
    auto fetch_snapshot = [&](int k) {
        const long long o = info->snap_off + (long long)k * info->slot + (warp * R * p.pitch + 2 * lane);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!(own >> r & 1)) continue;
            auto get = [&](int comp, int c) { cp_async_vec<2>(reinterpret_cast<float *>(&s_img(comp, 2, r)), p.snap[c] + o + (long long)r * p.pitch); };
            if constexpr (PSV) { get(0, 0); get(1, 2); }
            if constexpr (SH) get(0, 1);
        }
        cp_async_commit();
    };
    auto move_images = [&](bool in) {
        const long long io = info->img_off + (warp * R * p.pitch + 2 * lane);
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            if (!(own >> r & 1)) continue;
            auto move = [&](int comp, int c) {
                const long long at = io + (long long)r * p.pitch;
                if (in) {
                    s_img(comp, 0, r) = ld2(p.img[c], at);
                    s_img(comp, 1, r) = ld2(p.imgc[c], at);
                } else {
                    st2(p.img[c], at, s_img(comp, 0, r));
                    st2(p.imgc[c], at, s_img(comp, 1, r));
                }
            };
            if constexpr (PSV) { move(0, 0); move(1, 2); }
            if constexpr (SH) move(0, 1);
        }
    };
    // Finite check (fm:455-488, bm:417-450) of the owned cells.
    auto check = [&](int seq) {
        int code = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!(own >> r & 1)) continue;
            auto bad = [&](f2 x, int c) { code = max(code, max(bad_code(f2_lo(x), c), bad_code(f2_hi(x), c))); };
            if constexpr (PSV) { bad(U[r], p.code_base); bad(W[r], p.code_base + 2); }
            if constexpr (SH) bad(V[r], p.code_base + 1);
        }
        code = __reduce_max_sync(FULL, code);
        if (lane == 0 && code > 0) {
            atomicMax(p.flags + info->shot, code);
            atomicMin(p.fail_seq + info->shot, seq);
            info->bad = 1;
        }
    };

    // the state of the owned cells to store[] + at
    auto store_state = [&](long long at) {
        const long long so = state_at(my_row0(), my_col()) + at;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!(own >> r & 1)) continue;
            store_row(r, so + (long long)r * p.pitch, p.store);
        }
    };

    // ---- time loop
    publish_sig();
    int it = p.it0, checks = 0, blk = 0;
    bool check_last = false;  // the block before ended at a checked step
    int next_check = p.it1;   // next checked step, p.it1: none left
    if (p.check_interval > 0) {
        const int d = it % p.check_interval;
        next_check = d == 0 ? it : p.check_interval - d < p.it1 - it ? it + p.check_interval - d : p.it1;
    }
    // the next imaging step and its m; p.it1 or later: none left.  (Found by a division
    // per step, with the slot's offset from the window's: 500 cycles per step, on warps
    // without a cell to store too.)
    int img_it = p.it1, img_m = 0;
    if (p.isnap > 0) {
        if constexpr (DIR == 0) {
            img_m = max(p.snap_lo, it / p.isnap + (it % p.isnap != 0));
            if (img_m <= p.snap_hi && (long long)img_m * p.isnap < p.it1) img_it = img_m * p.isnap;
        } else {
            img_m = min(p.snap_hi, (p.nt - 1 - it) / p.isnap);
            if (img_m >= p.snap_lo) img_it = p.nt - 1 - img_m * p.isnap;
        }
    }
    if (DIR == 1 && p.img_chip) {
        move_images(true);
        if (img_it < p.it1) fetch_snapshot(img_m - p.snap_base);
    }
    while (it < p.it1) {
        // steps of this block: up to H, ending at a checked step
        int n = min(RES_HALO, p.it1 - it);
        const bool made = check_last;
        n = min(n, next_check - it + 1);
        // injection values of the block
        const int n_inj = s_ip[RT];
        for (int k = threadIdx.x; k < n * n_inj; k += 32 * NW) {
            const int s = k / n_inj, e = k - s * n_inj, id = s_inj[e].y;
            auto stage = [&](int comp, int c) {
                const float *src;
                if constexpr (DIR == 0) src = p.wav[c] + (size_t)id * p.nt + (it + s);
                else src = p.obs[c] + (size_t)(p.nt - 1 - (it + s)) * p.nrec_total + id;
                cp_async_vec<1>(s_val() + ((size_t)s * NC + comp) * p.max_inj + e, src);
            };
            if constexpr (PSV) { stage(0, 0); stage(1, 2); }
            if constexpr (SH) stage(0, 1);
        }
        cp_async_commit();
        if (blk > 0) {
            // exchange blk: send the frame, collect the halo
            const unsigned tag = p.tag0 + (unsigned)blk;
            const int row0 = my_row0(), col = my_col(), nx = info->nx;
            uint4 *const box = p.outbox + (size_t)(blk & 1) * L::BOX;  // this exchange's outbox of CTA 0
            if (own) {
                const bool side = lane < RES_HALO || lane >= 32 - RES_HALO;
                const int ol = lane - RES_HALO / 2;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int rr = warp * R + r;
                    if (!(own >> r & 1) || !(side || rr < 2 * RES_HALO || rr >= RT - 2 * RES_HALO)) continue;
                    uint4 *q = box + (size_t)blockIdx.x * p.box_stride + (rr - RES_HALO) * (L::NP * L::OLN) + ol;
                    if (!RTM_DBG_OK(q, 16) || !RTM_DBG_OK(q + (L::NP - 1) * L::OLN, 16)) continue;
                    // packet k: pair k and one value of the pairs left over
                    if constexpr (PSV) {
                        st_packet(q, U[r], f2_lo(W[r]), tag);
                        st_packet(q + L::OLN, XX[r], f2_hi(W[r]), tag);
                        st_packet(q + 2 * L::OLN, ZZ[r], f2_lo(XZ[r]), tag);
                        st_packet(q + 3 * L::OLN, 0ull, f2_hi(XZ[r]), tag);
                    } else {
                        st_packet(q, V[r], f2_lo(YZ[r]), tag);
                        st_packet(q + L::OLN, YX[r], f2_hi(YZ[r]), tag);
                    }
                }
            }
            // Halo packets, spread over the warps: a unit is one packet of one whole
            // halo row (32 lanes), or of the 2 + 2 side pairs of 8 rows.
            float *const stage = reinterpret_cast<float *>(sm0 + L::VEL);  // [halo pair][NF]
            const int ntj = info->ntj, col0 = info->col0, trow0 = info->row0 - RES_HALO;
            // lane part of a source: producer tile column and its lane
            auto lane_part = [&](int ln) -> int {
                const int j = col0 - RES_HALO + 2 * ln;
                if ((unsigned)j >= (unsigned)p.nz) return INT_MIN;
                int pl = ln - RES_HALO / 2, d = 0;
                if (pl < 0) { pl += L::OLN; d = -p.box_stride; }
                else if (pl >= L::OLN) { pl -= L::OLN; d = p.box_stride; }
                return d + pl;
            };
            const uint4 *const me = box + (size_t)blockIdx.x * p.box_stride;
            constexpr int FU = 2 * RES_HALO * L::NP, FP = (FU + NW - 1) / NW;              // whole-row units, per warp
            constexpr int G = 32 / RES_HALO, SU = (L::ORW * L::NP + G - 1) / G, SP = (SU + NW - 1) / NW;  // side units
            const int sl = lane % RES_HALO, sln = sl < RES_HALO / 2 ? sl : sl + L::OLN;
            const int lp = lane_part(lane), slp = lane_part(sln);
            const uint4 *src[FP + SP];
            Packet pk[FP + SP];
            unsigned pending = 0;
#pragma unroll
            for (int k = 0; k < FP + SP; ++k) {
                bool in;
                if (k < FP) {
                    const int u = k * NW + warp, pn = u % L::NP, hr = u / L::NP;  // hr: 0 .. 2H-1
                    const bool up = hr < RES_HALO;
                    const int i = trow0 + (up ? hr : hr + L::ORW), pr = up ? L::ORW - RES_HALO + hr : hr - RES_HALO;
                    in = (FU % NW == 0 || u < FU) && lp != INT_MIN && (unsigned)i < (unsigned)nx;
                    src[k] = me + ((up ? -ntj : ntj) * p.box_stride + (pr * L::NP + pn) * L::OLN + lp);
                } else {
                    const int m = ((k - FP) * NW + warp) * G + lane / RES_HALO, pr = m / L::NP;  // owned row; packet m % NP
                    in = m < L::ORW * L::NP && slp != INT_MIN && trow0 + RES_HALO + pr < nx;
                    src[k] = me + (m * L::OLN + slp);
                }
                pk[k].pair = pk[k].rest = 0ull;
                if (in && RTM_DBG_OK(src[k], 16)) pending |= 1u << k;
            }
            // All packets are asked for at once, those still missing again together.
            // (Polling with three lanes first, to spare L2 the traffic, was slower:
            // 9,058 against 8,517 cycles per block on a 301 x 151 shot.)
            // A check that the last block made is settled here too: every tile of the
            // shot has sent its count by now, and nothing has been put out since.  (A
            // wait of its own after the check took 6,000 cycles, most of them for the
            // fence and the chain of three L2 round trips.)  Checks alternate between
            // two counters, so a tile that is already past the next check cannot be
            // mistaken for one that has made this one.
            bool ask = made && threadIdx.x == 0;
            const unsigned long long *const arrive = p.arrive + 2 * info->shot + (checks & 1);
#ifdef RTM_BOUNDS_CHECK
            int n = p.polls0;
#else
            int n = 0;  // a constant: from an argument, 1001 x 501 SH took 1.77 ms instead of 1.72 (another loop, fewer spills)
#endif
            for (;;) {
                unsigned long long seen = 0;
                if (ask) seen = ld_relaxed(arrive);
#pragma unroll
                for (int k = 0; k < FP + SP; ++k)
                    if (pending >> k & 1) ld_packet(pk[k], src[k]);
                if (ask && (unsigned)seen == (unsigned)((checks + 1) / 2 * info->tiles)) {
                    ask = false;
                    if (seen >> 32) info->leave = 2;
                }
#pragma unroll
                for (int k = 0; k < FP + SP; ++k)
                    if (pk[k].tag() == tag) pending &= ~(1u << k);
                if (!pending && !ask) break;
                if (++n >= RES_SPIN_LIMIT || ((n & 1023) == 1023 && ld_acquire(p.err) != 0)) {
                    atomicExch(p.err, 1);
                    atomicExch(p.err + 1, 1);
                    info->leave = 1;
                    break;
                }
            }
#pragma unroll
            for (int k = 0; k < FP + SP; ++k) {
                int cell, pn;
                if (k < FP) {
                    const int u = k * NW + warp;
                    if (FU % NW && u >= FU) continue;
                    cell = u / L::NP * 32 + lane;
                    pn = u % L::NP;
                } else {
                    const int m = ((k - FP) * NW + warp) * G + lane / RES_HALO;
                    if (m >= L::ORW * L::NP) continue;
                    cell = 2 * RES_HALO * 32 + m / L::NP * RES_HALO + sl;
                    pn = m % L::NP;
                }
                // a cell's staged pairs: the packets' pairs, then the pairs they carry in halves
                float *q = stage + cell * L::NF;
                if (pn < L::NPAIR) *reinterpret_cast<f2 *>(q + 2 * pn) = pk[k].pair;
                if (pn < L::NF - 2 * L::NPAIR) q[2 * L::NPAIR + pn] = f2_lo(pk[k].rest);
            }
            __syncthreads();
            if (info->leave) break;
            const bool ci = (unsigned)col < (unsigned)p.nz;
            const unsigned in = rows_in(row0, nx);
            const bool hl = lane < RES_HALO / 2 || lane >= 32 - RES_HALO / 2;
            const unsigned sbase = (unsigned)__cvta_generic_to_shared(stage);
            const int slane = 2 * RES_HALO * 32 + (lane < RES_HALO / 2 ? lane : lane - L::OLN);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int rr = warp * R + r;
                const bool hr = rr < RES_HALO || rr >= RT - RES_HALO;
                const bool get = (hl || hr) && ci && (in >> r & 1);
                const int cell = hr ? (rr < RES_HALO ? rr : rr - L::ORW) * 32 + lane : slane + (rr - RES_HALO) * RES_HALO;
                const unsigned q = sbase + cell * (L::NF * 4);
                if constexpr (PSV) {
                    lds_if(U[r], q, get); lds_if(XX[r], q + 8, get); lds_if(ZZ[r], q + 16, get);
                    lds_if(W[r], q + 24, get); lds_if(XZ[r], q + 32, get);
                }
                if constexpr (SH) { lds_if(V[r], q, get); lds_if(YX[r], q + 8, get); lds_if(YZ[r], q + 16, get); }
            }
            __syncthreads();
            publish_sig();
        }
        cp_async_wait<0>();
        __syncthreads();
        for (int s = 0; s < n; ++s, ++it) {
            if (kind >= 2) velocity(std::true_type{});
            else velocity(std::false_type{});
            if (DIR == 0 ? sources : points == 2) inject_list(s);
            else if (DIR == 1 && points == 1) inject_table(s);
            publish_vel();
            __syncthreads();
            if (kind == 0) stress(std::integral_constant<int, 0>{});
            else if (kind == 1) stress(std::integral_constant<int, 1>{});
            else if (kind == 2) stress(std::integral_constant<int, 2>{});
            else stress(std::integral_constant<int, 3>{});
            publish_sig();
            const int t = DIR == 0 ? it : p.nt - 1 - it;
            if constexpr (DIR == 0) {
                if (points) record(t);
                if (p.keep_every && (it + 1 - p.it0) % p.keep_every == 0 && it + 1 < p.nt)
                    store_state(((it + 1 - p.it0) / p.keep_every - 1) * p.keep);
            }
            if (it == img_it) {
                snapshot(img_m - p.snap_base);
                img_m += DIR == 0 ? 1 : -1;
                img_it = (DIR == 0 ? img_m <= p.snap_hi : img_m >= p.snap_lo) && p.isnap < p.it1 - it ? it + p.isnap : p.it1;
                // the next one's copies are under way while the steps up to it run
                if (DIR == 1 && p.img_chip && img_it < p.it1) fetch_snapshot(img_m - p.snap_base);
            }
            if (it == next_check) check(it + 1);
            __syncthreads();
        }
        ++blk;
        check_last = it == next_check + 1;
        if (check_last) {
            ++checks;
            if (threadIdx.x == 0)
                atomicAdd(p.arrive + 2 * info->shot + (checks & 1), info->bad ? (1ull << 32) + 1 : 1ull);
            next_check = p.check_interval < p.it1 - next_check ? next_check + p.check_interval : p.it1;
        }
    }
    cp_async_wait<0>();
    if (DIR == 1 && p.img_chip) move_images(false);
    // final state of the owned cells; a shot that stopped inside a segment leaves none
    if (p.store[PSV ? F_U : F_V] && !(DIR == 0 && p.keep_every) && !(p.segment && info->leave == 2 && it < p.it1)) store_state(0);
}

template <int DIR, int MODE, int R, int NW>
__global__ void __launch_bounds__(32 * NW, res_ctas<MODE, R, NW>()) resident_kernel(const ResParams p) {
    resident_body<DIR, MODE, R, NW>(p);
}

// Both wave types: they never read each other's fields, so each has tiles of its
// own, with its own rows per lane; the finite checks stop them together.  (One
// tile for both takes 128 registers at R 2: 86 against 97 Gcell/s on a full chip,
// and 1.85 against 1.07 us per step on 72 x 56.)
template <int DIR, int RP, int RS, int NW>
__global__ void __launch_bounds__(32 * NW, res_ctas<1, RP, NW>() < res_ctas<2, RS, NW>() ? res_ctas<1, RP, NW>() : res_ctas<2, RS, NW>())
resident_both_kernel(const ResParams p) {
    if (p.tiles[p.tile0 + blockIdx.x].w == 0) resident_body<DIR, 1, RP, NW>(p);
    else resident_body<DIR, 2, RS, NW>(p);
}

}  // namespace rtm

// Resident interval kernel: a whole forcing interval of a network whose state
// fits in the shared memory of the GPU's SMs, in one cooperative launch.
//
// Each CTA (one per SM) owns a tile of consecutive catchments, the levees in
// them and the bifurcation paths that start in them, and holds their
// parameters, topology and state in shared memory from the first sub-step to
// the last.  In the breadth-first order 96-99 % of the neighbours of a
// 400-1700-cell tile lie in the tile itself: they meet at the CTA's barrier
// after each of the three phases (momentum, limit rate, stage with levees).
//
// What crosses tiles -- a cell's fluxes and limit rate, read by the tile of
// its downstream cell; its water surface and limit rate, read by the tiles of
// its upstream cells; a path's end state, limit rates and sums -- goes through
// L2 as words of 32 value bits and a 32-bit epoch, written and read whole.  A
// reader polls the word until it carries the epoch of the sub-step, so a value
// arrives with its own flag, with no fence and no grid barrier.  Between the
// phases all threads together fetch the values that the tile needs from
// others (its upstream cells elsewhere are one contiguous range) into shared
// memory, one round trip for all of them.  No word is overwritten early,
// because every word's next value depends on its reader's answer to this one:
//
//   fluxes of c (read by its downstream cell d's tile in the limit and stage
//     phases) are written again after c has read d's next water surface, which
//     d publishes after its stage;
//   surface and limit rate of d likewise wait for the fluxes of its upstream
//     cells, whose threads have read the old ones before;
//   a path's sums wait for the next state of its second end, which the end
//     publishes after reading them; the rates and states of the ends wait for
//     the path's next sums, which the path computes after its stage.
//
// A phase needs other tiles' values of earlier phases only, so no wait depends
// on a thread of its own warp, and all CTAs are co-resident (cooperative
// launch), so every wait ends.  Each is still bounded, in polls and not in time:
// a process that is swapped off a shared GPU loses time but makes no polls.
// After them CMF_STATUS_SYNC_TIMEOUT and the abort word are set and every CTA
// leaves.
#pragma once

#include "cmf_device.cuh"

namespace cmf {

// REAL-typed per-cell fields of a tile in shared memory
enum ResidentField {
    RF_WIDTH = 0, RF_LEN, RF_BANK, RF_NRIV, RF_NFLD, RF_ELEV, RF_DX, RF_AREA, RF_RUNOFF,  // static
    RF_ROUT, RF_FOUT, RF_RDEP, RF_FDEP, RF_RCSD, RF_FCSD, RF_FCSA,                        // state
    RF_QR, RF_QF, RF_LR,                                                                  // of the sub-step
    kResidentFields
};
// REAL-typed fields per level of an own path
enum PathLevelField { PL_SILL = 0, PL_WIDTH, PL_NRIV, PL_FLUX, PL_DEPTH, kPathLevelFields };
// of a path end: the path's summed fluxes and, where it is elsewhere, the
// other end's limit rate
enum PathEndField { PE_SUM = 0, PE_RAW, PE_RATE, kPathEndFields };
// of a levee: its parameters, its marks and its protected depth
enum LeveeTileField {
    LF_CROWN = 0, LF_FRAC, LF_BASE, LF_SBASE, LF_SCROWN, LF_STOP, LF_SFIRST, LF_DW, LF_DIST, LF_PDEP,
    kLeveeTileFields
};
enum DamTileField { DF_CONS = 0, DF_ADJ, DF_EMERG, DF_NORM, DF_QADJ, DF_FLOOD, kDamTileFields };
// of an upstream cell in another tile
enum HaloField { HF_QR = 0, HF_QF, HF_LR, kHaloFields };
constexpr int kPathLanes = 8;  // lanes per path: one per level (kMaxBifLevels)
// tile-local bits of a cell's flag byte
constexpr uint8_t kRemoteDown = 64, kRemoteUp = 128;

// The most path ends, own paths, levees, dams and upstream cells elsewhere of
// any tile.
struct TileCounts {
    int ends, paths, levees, dams, halo;
};

// A tile's shared memory, sized for those counts: offsets in bytes, computed
// once per plan.
struct ResidentArgs {
    int tile;          // cells per tile
    TileCounts most;
    int fixed_n;       // > 0: the sub-step count, otherwise the CFL decides
    unsigned polls;    // polls after which a wait gives up
    int leave_step;    // sub-step at which the last tile leaves, for the test of that (-1: none)
    int o_rows;        // 0: the floodplain rows stay in L2
    int o_path, o_ends, o_levee, o_dam, o_halo, o_int, o_slot, o_flag;
    int bytes;
};

inline void resident_layout(ResidentArgs& a, int real, int K, int L, bool rows)
{
    const TileCounts& m = a.most;
    int o = 8 * (2 * a.tile + m.levees + m.dams) + a.tile * kResidentFields * real;
    a.o_rows = rows ? o : 0;
    if (rows) o += a.tile * K * real;
    a.o_path = o;
    o += m.paths * (kPathLevelFields * L + 1) * real;
    a.o_ends = o;
    o += m.ends * kPathEndFields * real;
    a.o_levee = o;
    o += m.levees * kLeveeTileFields * real;
    a.o_dam = o;
    o += m.dams * kDamTileFields * real;
    a.o_halo = o;
    o += m.halo * kHaloFields * real;
    a.o_int = o;
    o += 4 * (4 * a.tile + 1 + 2 * m.ends + 5 * m.paths + m.levees);
    a.o_slot = o;
    o += 2 * a.tile * ((m.levees > 0) + (m.dams > 0));
    a.o_flag = o;
    a.bytes = (o + a.tile + 15) / 16 * 16;
}

template <typename REAL>
constexpr int resident_threads() { return sizeof(REAL) == 4 ? 1024 : 512; }

template <typename REAL>
struct Tile {
    int t0, count, stride;  // first cell, cells, capacity
    TileCounts most;
    double *rs, *fs;        // storages
    double *ps, *rti;       // protected storage per levee, total inflow per dam
    REAL* f;                // cell fields
    const REAL* rows;       // [K][stride], or null
    REAL *pl, *plen;        // own paths: by level, lengths
    REAL *pe, *lf, *df, *hf;
    int *dn, *c0, *c1;
    int* end_of;            // [tile + 1] first path end of each cell
    int *end, *end_other;   // path end code (2 path + end); local cell of the other end, -1 elsewhere
    int *path, *path_a, *path_b, *path_xa, *path_xb;  // own paths; cells and entries of their ends (-1 elsewhere)
    int* levee_cell;
    uint16_t *levee_of, *dam_of;  // per cell
    uint8_t* fl;
    __device__ REAL& at(int field, int j) const { return f[field * stride + j]; }
    __device__ REAL& end_at(int field, int x) const { return pe[field * most.ends + x]; }
    __device__ REAL& levee_at(int field, int s) const { return lf[field * most.levees + s]; }
    __device__ REAL& dam_at(int field, int s) const { return df[field * most.dams + s]; }
    __device__ REAL& halo_at(int field, int x) const { return hf[field * most.halo + x]; }
    __device__ bool has(int cell) const { return (unsigned)(cell - t0) < (unsigned)count; }
};

template <typename REAL>
__device__ __forceinline__ Tile<REAL> tile_of(const Dev<REAL>& v, const ResidentArgs& a, unsigned char* smem)
{
    Tile<REAL> t;
    t.stride = a.tile;
    t.t0 = blockIdx.x * a.tile;
    t.count = min(a.tile, (int)v.N - t.t0);
    t.most = a.most;
    t.rs = reinterpret_cast<double*>(smem);
    t.fs = t.rs + a.tile;
    t.ps = t.fs + a.tile;
    t.rti = t.ps + a.most.levees;
    t.f = reinterpret_cast<REAL*>(t.rti + a.most.dams);
    t.rows = a.o_rows ? reinterpret_cast<const REAL*>(smem + a.o_rows) : nullptr;
    t.pl = reinterpret_cast<REAL*>(smem + a.o_path);
    t.plen = t.pl + a.most.paths * kPathLevelFields * v.L;
    t.pe = reinterpret_cast<REAL*>(smem + a.o_ends);
    t.lf = reinterpret_cast<REAL*>(smem + a.o_levee);
    t.df = reinterpret_cast<REAL*>(smem + a.o_dam);
    t.hf = reinterpret_cast<REAL*>(smem + a.o_halo);
    t.dn = reinterpret_cast<int*>(smem + a.o_int);
    t.c0 = t.dn + a.tile;
    t.c1 = t.c0 + a.tile;
    t.end_of = t.c1 + a.tile;
    t.end = t.end_of + a.tile + 1;
    t.end_other = t.end + a.most.ends;
    t.path = t.end_other + a.most.ends;
    t.path_a = t.path + a.most.paths;
    t.path_b = t.path_a + a.most.paths;
    t.path_xa = t.path_b + a.most.paths;
    t.path_xb = t.path_xa + a.most.paths;
    t.levee_cell = t.path_xb + a.most.paths;
    t.levee_of = reinterpret_cast<uint16_t*>(smem + a.o_slot);
    t.dam_of = t.levee_of + (a.most.levees > 0 ? a.tile : 0);
    t.fl = smem + a.o_flag;
    return t;
}

// ---------------------------------------------------------------------------
// waits
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned load_acquire_u32(const unsigned* p)
{
    unsigned x;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
    return x;
}
__device__ __forceinline__ void store_release_u32(unsigned* p, unsigned x)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}
__device__ __forceinline__ unsigned long long load_word(const unsigned long long* p)
{
    unsigned long long x;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
    return x;
}
__device__ __forceinline__ void store_word(unsigned long long* p, unsigned long long x)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}

// Polls of a wait, each an L2 round trip (some 0.3-0.7 us): seconds of a wait
// that takes microseconds.
constexpr unsigned kWaitPolls = 1u << 22;
constexpr unsigned kPollsPerCheck = 64;  // between two looks at the abort word

// A wait's look at how it stands after `spin` polls of at most `polls`: true
// when it has to give up, because it has used them or another one has.  `quit`
// tells the CTA.
__device__ __forceinline__ bool wait_over(int* ctl, int* status, unsigned spin, unsigned polls, int* quit)
{
    if (!*reinterpret_cast<volatile int*>(ctl + kCtlAbort)) {
        if (spin < polls) return false;
        atomicOr(status, CMF_STATUS_SYNC_TIMEOUT);
        atomicExch(ctl + kCtlAbort, 1);
    }
    *reinterpret_cast<volatile int*>(quit) = 1;
    return true;
}

// Whether any thread of the CTA has seen a wait give up (a CTA barrier).
__device__ __forceinline__ bool cta_quits(const int* quit)
{
    return __syncthreads_or(*reinterpret_cast<const volatile int*>(quit));
}

// All tiles meet (once per interval, for the sub-step count); true: leave.
__device__ __forceinline__ bool tiles_meet(unsigned* flags, int* ctl, int* status, int tiles, unsigned polls,
                                           int* quit)
{
    __syncthreads();
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) store_release_u32(flags + blockIdx.x, 1u);
        for (int q = threadIdx.x; q < tiles; q += 32) {
            for (unsigned spin = 1; load_acquire_u32(flags + q) == 0; ++spin)
                if (spin % kPollsPerCheck == 0 && wait_over(ctl, status, spin, polls, quit)) break;
        }
    }
    return cta_quits(quit);
}

// What a CTA needs to wait for a word.
struct Wait {
    int *ctl, *status, *quit;
    unsigned epoch, polls;
};

// The value bits of a word whose first read gave x, once it carries the epoch.
__device__ __forceinline__ unsigned await_word(const unsigned long long* p, unsigned long long x, const Wait& w)
{
    if ((unsigned)(x >> 32) != w.epoch) {
        for (unsigned spin = 1;; ++spin) {
            x = load_word(p);
            if ((unsigned)(x >> 32) == w.epoch) break;
            if (spin % kPollsPerCheck == 0 && wait_over(w.ctl, w.status, spin, w.polls, w.quit)) break;
        }
    }
    return (unsigned)x;
}

// A value in words of 32 bits of it and the epoch: one for a float, two for a
// double.
template <typename REAL>
__device__ __forceinline__ void post(unsigned long long* p, long i, REAL x, unsigned epoch)
{
    const unsigned long long e = (unsigned long long)epoch << 32;
    if constexpr (sizeof(REAL) == 4) {
        store_word(p + i, e | __float_as_uint(x));
    } else {
        const unsigned long long b = __double_as_longlong(x);
        store_word(p + 2 * i, e | (b & 0xffffffffull));
        store_word(p + 2 * i + 1, e | (b >> 32));
    }
}

// COUNT consecutive values, their words read together.
template <int COUNT, typename REAL>
__device__ __forceinline__ void fetch(const unsigned long long* p, long i, const Wait& w, REAL (&out)[COUNT])
{
    constexpr int W = sizeof(REAL) / 4;
    const unsigned long long* q = p + i * W;
    unsigned long long x[COUNT * W];
#pragma unroll
    for (int k = 0; k < COUNT * W; ++k) x[k] = load_word(q + k);
#pragma unroll
    for (int k = 0; k < COUNT; ++k) {
        if constexpr (W == 1) {
            out[k] = __uint_as_float(await_word(q + k, x[k], w));
        } else {
            const unsigned long long lo = await_word(q + 2 * k, x[2 * k], w);
            const unsigned long long hi = await_word(q + 2 * k + 1, x[2 * k + 1], w);
            out[k] = __longlong_as_double((long long)(hi << 32 | lo));
        }
    }
}

template <typename REAL>
__device__ __forceinline__ REAL fetch(const unsigned long long* p, long i, const Wait& w)
{
    REAL x[1];
    fetch(p, i, w, x);
    return x[0];
}

// The rarely read fields of a cell, in the tile (momentum_rates).
template <typename REAL>
struct TileRare {
    const Tile<REAL>& t;
    int j;
    __device__ REAL river_store() const { return (REAL)t.rs[j]; }
    __device__ REAL protected_store() const { return (REAL)t.ps[t.levee_of[j]]; }
    __device__ REAL protected_depth() const { return t.levee_at(LF_PDEP, t.levee_of[j]); }
    __device__ DamRule<REAL> dam_rule() const
    {
        const int s = t.dam_of[j];
        return {t.dam_at(DF_CONS, s), t.dam_at(DF_ADJ, s), t.dam_at(DF_EMERG, s),
                t.dam_at(DF_NORM, s), t.dam_at(DF_QADJ, s), t.dam_at(DF_FLOOD, s)};
    }
    __device__ REAL dam_inflow() const { return (REAL)t.rti[t.dam_of[j]] + t.at(RF_RUNOFF, j); }
};

// A cell's floodplain profile on a row in shared memory or, with its first
// two levels loaded ahead, in L2.
template <typename REAL>
struct RowProfile {
    const REAL* row;
    int step;   // 1: in L2
    int K;
    REAL ca;
    bool ahead;  // whether they are
    REAL d0, d1;
    __device__ REAL area() const { return ca; }
    __device__ FillLevel<REAL> walk(REAL S, REAL bank, REAL width, REAL len, REAL dw) const
    {
        FillLevel<REAL> f{0, bank, REAL(0), REAL(0)};
        REAL w_lo = width;
        int l = 0;
        if (ahead) {
            if (!fill_layer(f, w_lo, 0, d0, S, width, len, dw)) return f;
            if (!fill_layer(f, w_lo, 1, d1, S, width, len, dw)) return f;
            l = 2;
        }
        for (; l < K; ++l)
            if (!fill_layer(f, w_lo, l, row[l * step], S, width, len, dw)) break;
        return f;
    }
};

// Level fields of the tile's own path s.
template <typename REAL>
struct TilePathLevels {
    const Tile<REAL>& t;
    int s, L;
    __device__ REAL& at(int field, int l) const { return t.pl[(field * t.most.paths + s) * L + l]; }
    __device__ REAL sill(int l) const { return at(PL_SILL, l); }
    __device__ REAL width(int l) const { return at(PL_WIDTH, l); }
    __device__ REAL manning(int l) const { return at(PL_NRIV, l); }
    __device__ REAL flux(int l) const { return at(PL_FLUX, l); }
    __device__ REAL depth(int l) const { return at(PL_DEPTH, l); }
};

// State of local cell j as an end of a path (path_end_state).
template <typename REAL, bool RES, bool LEV>
__device__ __forceinline__ void tile_end_state(const Tile<REAL>& t, int j, REAL& eta, REAL& peta, REAL& store)
{
    const uint8_t fl = t.fl[j];
    const REAL elev = t.at(RF_ELEV, j);
    eta = t.at(RF_RDEP, j) + (elev - t.at(RF_BANK, j));
    const bool lev_cell = LEV && (fl & CMF_CELL_LEVEE);
    peta = lev_cell ? smin(elev + t.levee_at(LF_PDEP, t.levee_of[j]), eta) : eta;
    const REAL held = (REAL)t.rs[j] + (REAL)t.fs[j];
    store = (RES && (fl & CMF_CELL_RESERVOIR)) ? held
                                               : held + (lev_cell ? (REAL)t.ps[t.levee_of[j]] : REAL(0));
}

// Publishes the state of local cell j at the start of the sub-step of `epoch`
// to the tiles that read it.
template <typename REAL, bool RES, bool LEV, bool BIF>
__device__ __forceinline__ void publish_state(const Dev<REAL>& v, const Tile<REAL>& t, int j, unsigned epoch)
{
    const uint8_t fl = t.fl[j];
    if (fl & kRemoteUp) post(v.xeta, t.t0 + j, t.at(RF_RDEP, j) + (t.at(RF_ELEV, j) - t.at(RF_BANK, j)), epoch);
    if (BIF && (fl & CMF_CELL_BIFURCATION)) {
        for (int b = t.end_of[j]; b < t.end_of[j + 1]; ++b) {
            const int e = t.end[b];
            if (!(e & 1) || t.end_other[b] >= 0) continue;  // the path is this tile's own
            REAL eta, peta, store;
            tile_end_state<REAL, RES, LEV>(t, j, eta, peta, store);
            const long x = 3L * (e >> 1);
            post(v.xend, x, eta, epoch);
            post(v.xend, x + 1, peta, epoch);
            post(v.xend, x + 2, store, epoch);
        }
    }
}

// ---------------------------------------------------------------------------
// phases, one cell or path each
// ---------------------------------------------------------------------------
template <typename REAL, bool RES, bool LEV>
__device__ __forceinline__ void resident_momentum(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w, int j,
                                                  REAL dt, bool diag)
{
    const int i = t.t0 + j;
    const uint8_t fl = t.fl[j];
    const int dn = t.dn[j], d = dn - t.t0;
    MomentumCell<REAL> c;
    c.width = t.at(RF_WIDTH, j);
    c.len = t.at(RF_LEN, j);
    c.bank_h = t.at(RF_BANK, j);
    c.n_riv = t.at(RF_NRIV, j);
    c.n_fld = t.at(RF_NFLD, j);
    c.elev = t.at(RF_ELEV, j);
    c.dx = t.at(RF_DX, j);
    c.q_riv = t.at(RF_ROUT, j);
    c.q_fld = t.at(RF_FOUT, j);
    c.h_riv = t.at(RF_RDEP, j);
    c.h_fld = t.at(RF_FDEP, j);
    c.hr_before = t.at(RF_RCSD, j);
    c.hf_before = t.at(RF_FCSD, j);
    c.af_before = t.at(RF_FCSA, j);
    c.s_fld = (REAL)t.fs[j];
    if (!(fl & kRemoteDown)) {
        c.elev_dn = t.at(RF_ELEV, d);
        c.eta_dn = (fl & CMF_CELL_MOUTH) ? c.elev : t.at(RF_RDEP, d) + (c.elev_dn - t.at(RF_BANK, d));
    } else {
        c.elev_dn = RES && (fl & CMF_CELL_DAM_UPSTREAM) ? __ldg(v.celv + dn) : c.elev;
        c.eta_dn = fetch<REAL>(v.xeta, dn, w);
    }
    const TileRare<REAL> rare{t, j};
    const MomentumRates<REAL> r = momentum_rates<REAL, RES, LEV>(c, fl, dt, v.g, v.min_kin, rare);
    if (fl & kRemoteDown) {
        post(v.xflux, 2L * i, r.q_riv, w.epoch);
        post(v.xflux, 2L * i + 1, r.q_fld, w.epoch);
    }
    t.at(RF_QR, j) = r.q_riv;
    t.at(RF_QF, j) = r.q_fld;
    t.at(RF_RCSD, j) = r.h_riv;
    t.at(RF_FCSD, j) = r.h_fld;
    t.at(RF_FCSA, j) = r.a_fld;
    if (diag) momentum_diagnostics<REAL, RES, LEV>(v, c.elev, c.s_fld, fl, i, r.eta, rare);
}

// Own path s, one lane per level l in groups of kPathLanes; every lane of the
// warp comes here together, `live` for the levels that exist.
template <typename REAL, bool RES, bool LEV>
__device__ __forceinline__ void resident_path_momentum(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w,
                                                       int s, int lane_in_path, bool live, REAL dt)
{
    PathEnds<REAL> e{};
    REAL q = REAL(0), h = REAL(0);
    const TilePathLevels<REAL> lv{t, s, v.L};
    const int b = t.path_b[s];
    // a second end elsewhere: its three values by three lanes
    REAL far = REAL(0);
    if (b < 0 && lane_in_path < 3) far = fetch<REAL>(v.xend, 3L * t.path[s] + lane_in_path, w);
    e.eta_b = __shfl_sync(0xffffffffu, far, 0, kPathLanes);
    e.peta_b = __shfl_sync(0xffffffffu, far, 1, kPathLanes);
    e.store_b = __shfl_sync(0xffffffffu, far, 2, kPathLanes);
    tile_end_state<REAL, RES, LEV>(t, t.path_a[s], e.eta_a, e.peta_a, e.store_a);
    if (b >= 0) tile_end_state<REAL, RES, LEV>(t, b, e.eta_b, e.peta_b, e.store_b);
    const int l = lane_in_path;
    if (live) {
        const REAL top = smax(e.eta_a, e.eta_b);
        const REAL ptop = LEV ? smax(e.peta_a, e.peta_b) : top;
        q = path_level_flux<LEV>(lv, l, top, ptop, path_slope(e, t.plen[s]), v.g * dt, h);
    }
    // the sums in level order, as one thread per path forms them
    REAL sum = REAL(0);
    for (int k = 0; k < v.L; ++k) sum = sum + __shfl_sync(0xffffffffu, q, k, kPathLanes);
    const REAL rate = live ? path_rate(sum, e.store_a, e.store_b, dt) : REAL(0);
    const REAL moved = q * rate;
    REAL raw = REAL(0);
    for (int k = 0; k < v.L; ++k) raw = raw + __shfl_sync(0xffffffffu, moved, k, kPathLanes);
    if (!live) return;
    lv.at(PL_FLUX, l) = moved;
    lv.at(PL_DEPTH, l) = h;
    if (l == 0) {
        const int xa = t.path_xa[s], xb = t.path_xb[s];
        t.end_at(PE_SUM, xa) = sum * rate;
        t.end_at(PE_RAW, xa) = raw;
        if (xb >= 0) {
            t.end_at(PE_SUM, xb) = sum * rate;
            t.end_at(PE_RAW, xb) = raw;
        } else {
            const long x = 2L * t.path[s];
            post(v.xsum, x, sum * rate, w.epoch);
            post(v.xsum, x + 1, raw, w.epoch);
        }
    }
}

// Before the limit phase: the fluxes of the upstream cells elsewhere, and the
// sums of the paths that end here and belong to another tile.
template <typename REAL, bool BIF>
__device__ __forceinline__ void fetch_fluxes(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w, int halo0,
                                             int halo, int ends)
{
    for (int x = threadIdx.x; x < halo + ends; x += blockDim.x) {
        REAL q[2];
        if (x < halo) {
            fetch(v.xflux, 2L * (halo0 + x), w, q);
            t.halo_at(HF_QR, x) = q[0];
            t.halo_at(HF_QF, x) = q[1];
        } else if (BIF) {
            const int b = x - halo, e = t.end[b];
            if (!(e & 1) || t.end_other[b] >= 0) continue;
            fetch(v.xsum, 2L * (e >> 1), w, q);
            t.end_at(PE_SUM, b) = q[0];
            t.end_at(PE_RAW, b) = q[1];
        }
    }
}

// Before the stage: the limit rates of the upstream cells elsewhere and of
// the paths' other ends elsewhere.
template <typename REAL, bool BIF>
__device__ __forceinline__ void fetch_rates(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w, int halo0,
                                            int halo, int ends)
{
    for (int x = threadIdx.x; x < halo + ends; x += blockDim.x) {
        if (x < halo) {
            t.halo_at(HF_LR, x) = fetch<REAL>(v.xrate, halo0 + x, w);
        } else if (BIF) {
            const int b = x - halo;
            if (t.end_other[b] < 0) t.end_at(PE_RATE, b) = fetch<REAL>(v.xprate, t.end[b] ^ 1, w);
        }
    }
}

// Calls fold(qr, qf, lr) for the upstream cells of local cell j, in order; a
// trip reads kGather of them before it folds any, so that only the sums
// themselves form a chain (a mouth of the generated networks gathers a hundred
// cells, and its tile is then the one that the others wait for).  Those
// outside the tile follow those inside.
constexpr int kGather = 8;
template <bool RATE, typename REAL, typename Fold>
__device__ __forceinline__ void gather_upstream(const Tile<REAL>& t, int j, int halo0, Fold fold)
{
    auto run = [&](const REAL* qr, const REAL* qf, const REAL* lr, int n) {
        int b = 0;
        for (; b + kGather <= n; b += kGather) {
            REAL r[kGather], f[kGather], l[kGather];
#pragma unroll
            for (int k = 0; k < kGather; ++k) {
                r[k] = qr[b + k];
                f[k] = qf[b + k];
                l[k] = RATE ? lr[b + k] : REAL(0);
            }
#pragma unroll
            for (int k = 0; k < kGather; ++k) fold(r[k], f[k], l[k]);
        }
#pragma unroll 1
        for (; b < n; ++b) fold(qr[b], qf[b], RATE ? lr[b] : REAL(0));
    };
    const int c0 = t.c0[j], c1 = t.c1[j], t1 = t.t0 + t.count;
    if (c0 < t1) run(&t.at(RF_QR, c0 - t.t0), &t.at(RF_QF, c0 - t.t0), &t.at(RF_LR, c0 - t.t0), min(c1, t1) - c0);
    if (c1 > t1 && c1 > c0) {
        const int x = max(c0, t1);
        run(&t.halo_at(HF_QR, x - halo0), &t.halo_at(HF_QF, x - halo0), &t.halo_at(HF_LR, x - halo0), c1 - x);
    }
}

template <typename REAL, bool BIF>
__device__ __forceinline__ void resident_limit(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w, int j,
                                               REAL ts, int halo0)
{
    const uint8_t fl = t.fl[j];
    const REAL pos = fmax(t.at(RF_QR, j), (REAL)0.0) + fmax(t.at(RF_QF, j), (REAL)0.0);
    double og = (double)(pos * ts);
    gather_upstream<false>(t, j, halo0, [&](REAL qr, REAL qf, REAL) {
        const REAL neg = fmin(qr, (REAL)0.0) + fmin(qf, (REAL)0.0);
        og += (double)(-neg * ts);
    });
    const bool ends = BIF && (fl & CMF_CELL_BIFURCATION);
    if (ends) {
        for (int b = t.end_of[j]; b < t.end_of[j + 1]; ++b)
            og = outgoing_path(og, t.end_at(PE_SUM, b), t.end[b], ts);
    }
    const REAL lr = limit_rate_from((REAL)og, t.rs[j] + t.fs[j]);
    t.at(RF_LR, j) = lr;
    if (fl & (kRemoteDown | kRemoteUp)) post(v.xrate, t.t0 + j, lr, w.epoch);
    if (ends)
        for (int b = t.end_of[j]; b < t.end_of[j + 1]; ++b)
            if (t.end_other[b] < 0) post(v.xprate, t.end[b], lr, w.epoch);
}

template <typename REAL, bool RES, bool LEV, bool BIF>
__device__ __forceinline__ void resident_stage(const Dev<REAL>& v, const Tile<REAL>& t, const Wait& w, int j,
                                               REAL ts, int halo0, bool diag, bool want_fraction)
{
    const int i = t.t0 + j;
    const uint8_t fl = t.fl[j];
    const bool mouth = fl & CMF_CELL_MOUTH;
    const bool lev_cell = LEV && (fl & CMF_CELL_LEVEE);
    const bool res_cell = RES && (fl & CMF_CELL_RESERVOIR);
    const REAL qr = t.at(RF_QR, j), qf = t.at(RF_QF, j), lr_i = t.at(RF_LR, j);
    const double prot = lev_cell ? t.ps[t.levee_of[j]] : 0.0;
    // a row in L2 starts its way now where the cell was flooded
    RowProfile<REAL> prof{t.rows ? t.rows + j : v.tbl + (long)i * v.K, t.rows ? t.stride : 1, v.K,
                          t.at(RF_AREA, j), false, REAL(0), REAL(0)};
    if (!t.rows && t.fs[j] > 0.0 && v.K >= 2) {
        prof.ahead = true;
        prof.d0 = __ldg(prof.row);
        prof.d1 = __ldg(prof.row + 1);
    }
    double rin = 0.0, fin = 0.0, rti = 0.0;
    gather_upstream<true>(t, j, halo0, [&](REAL qr_up, REAL qf_up, REAL lr_up) {
        const REAL ur = limited_flux(qr_up, lr_up, lr_i);
        const REAL uf = limited_flux(qf_up, lr_up, lr_i);
        rin += (double)ur;
        fin += (double)uf;
        if (res_cell) rti += (double)(ur + uf);
    });
    REAL lr_dn = lr_i;
    if (!mouth && (qr < (REAL)0.0 || qf < (REAL)0.0))
        lr_dn = t.has(t.dn[j]) ? t.at(RF_LR, t.dn[j] - t.t0) : fetch<REAL>(v.xrate, t.dn[j], w);
    const REAL rout = (qr >= (REAL)0.0) ? qr * lr_i : qr * lr_dn;
    const REAL fout = (qf >= (REAL)0.0) ? qf * lr_i : qf * lr_dn;
    double gb = 0.0;
    if (BIF && (fl & CMF_CELL_BIFURCATION)) {
        for (int b = t.end_of[j]; b < t.end_of[j + 1]; ++b) {
            const int o = t.end_other[b];
            gb += path_net(t.end_at(PE_RAW, b), t.end[b], lr_i, o >= 0 ? t.at(RF_LR, o) : t.end_at(PE_RATE, b));
        }
    }

    const Continuity<double, REAL> c =
        continuity<double, REAL>(t.rs[j], t.fs[j], prot, (REAL)rin, rout, (REAL)fin, fout,
                                 BIF ? (REAL)gb : REAL(0), t.at(RF_RUNOFF, j), ts);
    const StageOut<double, REAL> s =
        flood_stage_of(c.total, t.at(RF_WIDTH, j), t.at(RF_LEN, j), t.at(RF_BANK, j), v.K, prof);

    t.at(RF_ROUT, j) = rout;
    t.at(RF_FOUT, j) = fout;
    t.rs[j] = s.rs;
    t.fs[j] = s.fs;
    t.at(RF_RDEP, j) = s.rdep;
    t.at(RF_FDEP, j) = s.fdep;
    if (want_fraction) v.ffr[i] = s.ffr;
    if (res_cell) t.rti[t.dam_of[j]] = rti;
    if (!lev_cell && !diag) publish_state<REAL, RES, LEV, BIF>(v, t, j, w.epoch + 1);
    if (diag) {
        if (!lev_cell) v.pdep[i] = s.fdep;
        if (v.rinf) v.rinf[i] = rin;
        if (v.finf) v.finf[i] = fin;
        if (v.lr) v.lr[i] = lr_i;
        if (v.gbif) v.gbif[i] = gb;
    }
    if (!isfinite(s.rs) || !isfinite(s.fs) || !isfinite(rout) || !isfinite(fout))
        atomicOr(v.status, CMF_STATUS_NONFINITE);
}

// Levee s of the tile, after the stage.
template <typename REAL, bool RES, bool LEV, bool BIF>
__device__ __forceinline__ void resident_levee(const Dev<REAL>& v, const Tile<REAL>& t, int s, int first,
                                               unsigned epoch, bool diag, bool want_fraction)
{
    const int j = t.levee_cell[s], i = t.t0 + j;
    LeveeState<double, REAL> lst;
    lst.rs = t.rs[j];
    lst.fs = t.fs[j];
    lst.rdep = REAL(0);
    lst.fdep = REAL(0);
    lst.ffr = REAL(0);
    const LeveeMarks<REAL, REAL> mk{t.levee_at(LF_SBASE, s), t.levee_at(LF_SCROWN, s), t.levee_at(LF_STOP, s),
                                    t.levee_at(LF_SFIRST, s), t.levee_at(LF_DW, s), t.levee_at(LF_DIST, s)};
    const REAL* row = t.rows ? t.rows + j : v.lpk_tbl + (long)(first + s) * v.K;
    const int step = t.rows ? t.stride : 1;
    const int regime = levee_by_marks<REAL>(
        lst, mk, t.at(RF_WIDTH, j), t.at(RF_BANK, j), t.at(RF_LEN, j), t.levee_at(LF_CROWN, s),
        t.levee_at(LF_FRAC, s), t.levee_at(LF_BASE, s), v.K, [=](int l) { return row[l * step]; },
        [&]() { return t.at(RF_FDEP, j); });
    t.ps[s] = lst.ps;
    t.levee_at(LF_PDEP, s) = lst.pdep;
    if (regime == kLeveeOvertopped) {
        t.fs[j] = lst.fs;
    } else if (regime == kLeveeFilling || regime == kLeveeWedge) {
        t.rs[j] = lst.rs;
        t.fs[j] = lst.fs;
        t.at(RF_RDEP, j) = lst.rdep;
        t.at(RF_FDEP, j) = lst.fdep;
        if (want_fraction) v.ffr[i] = lst.ffr;
    }
    if (!diag) publish_state<REAL, RES, LEV, BIF>(v, t, j, epoch);
}

// Statistics value of a cell after the sub-step (stat_value on the tile).
template <typename REAL>
__device__ __forceinline__ double resident_stat(const Dev<REAL>& v, const Tile<REAL>& t, int var, int j)
{
    const int i = t.t0 + j;
    switch (var) {
    case CMF_VAR_RIVER_OUTFLOW: return (double)t.at(RF_ROUT, j);
    case CMF_VAR_FLOOD_OUTFLOW: return (double)t.at(RF_FOUT, j);
    case CMF_VAR_TOTAL_OUTFLOW: return __dadd_rn((double)t.at(RF_ROUT, j), (double)t.at(RF_FOUT, j));
    case CMF_VAR_RIVER_DEPTH: return (double)t.at(RF_RDEP, j);
    case CMF_VAR_FLOOD_DEPTH: return (double)t.at(RF_FDEP, j);
    case CMF_VAR_FLOOD_FRACTION: return (double)v.ffr[i];
    case CMF_VAR_PROTECTED_DEPTH:
        return (double)((t.fl[j] & CMF_CELL_LEVEE) ? t.levee_at(LF_PDEP, t.levee_of[j]) : t.at(RF_FDEP, j));
    case CMF_VAR_RIVER_STORAGE: return t.rs[j];
    case CMF_VAR_FLOOD_STORAGE: return t.fs[j];
    case CMF_VAR_PROTECTED_STORAGE: return (t.fl[j] & CMF_CELL_LEVEE) ? t.ps[t.levee_of[j]] : 0.0;
    default: return 0.0;
    }
}

// First list position in [0, n) whose entry is >= x (ascending list).
__device__ __forceinline__ int first_at_least(const int* list, int n, int x)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (list[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// What k_resident_scan leaves at ctl[kCtlTileMax ..].
struct TileScan {
    TileCounts most;  // maxima over the tiles
    int irregular;    // not 0: the view's lists are not in the form below
    int cell_ends;    // the most path ends of a cell
    int stray;        // upstream ranges' cells less the cells that are upstream of one
};

// TileCounts of every tile (one block each) and the form of the lists that
// k_resident indexes by, once per plan.  A levee of the tile is found by
// bisection of the levee list and writes its cell's slot, so the list has to be
// strictly ascending, in range, and exactly the cells flagged as levee cells;
// a path end elsewhere answers only if its cell is flagged for bifurcation and
// is the one that the path names.  And a cell elsewhere posts to its downstream
// cell's tile, which waits for all cells of its upstream ranges there: so a mouth
// flows into itself, every other cell lies in the range of the one it flows into,
// after it, and the ranges of a tile hold no other cells.
// The sub-step kernels wait for nothing and ask for none of this.
template <typename REAL>
__global__ void __launch_bounds__(256) k_resident_scan(const Dev<REAL> v, int tile)
{
    __shared__ int own, dams, levees, bad, lo, hi, cell_ends, stray, beyond;
    const int t0 = blockIdx.x * tile, t1 = min(t0 + tile, (int)v.N);
    if (threadIdx.x == 0) { own = dams = levees = bad = hi = cell_ends = stray = beyond = 0; lo = INT32_MAX; }
    __syncthreads();
    for (int i = t0 + threadIdx.x; i < t1; i += blockDim.x) {
        const int c0 = v.up[i], c1 = upstream_end(v, (long)i);
        const uint8_t fl = v.flags[i];
        if (c0 < c1) {
            if (c0 <= i || c1 > v.N) bad = 1;
            atomicAdd(&stray, c1 - c0);
        }
        if (c0 < c1 && c1 > t1) {
            atomicMin(&lo, max(c0, t1));
            atomicMax(&hi, c1);
            atomicAdd(&beyond, c1 - max(c0, t1));
        }
        const int d = v.dn[i];
        if (((fl & CMF_CELL_MOUTH) != 0) != (d == i)) bad = 1;
        if (d != i) {
            if (d < 0 || d >= v.N || i < v.up[d] || i >= upstream_end(v, (long)d)) bad = 1;
            atomicSub(&stray, 1);
        }
        if ((v.features & CMF_FEAT_RESERVOIR) && (fl & CMF_CELL_RESERVOIR)) atomicAdd(&dams, 1);
        if ((v.features & CMF_FEAT_LEVEE) && (fl & CMF_CELL_LEVEE)) atomicAdd(&levees, 1);
        if ((v.features & CMF_FEAT_BIFURCATION) && v.bptr[i] < v.bptr[i + 1]) {
            if (!(fl & CMF_CELL_BIFURCATION)) bad = 1;
            atomicMax(&cell_ends, v.bptr[i + 1] - v.bptr[i]);
        }
    }
    if (v.features & CMF_FEAT_BIFURCATION)
        for (int x = v.bptr[t0] + threadIdx.x; x < v.bptr[t1]; x += blockDim.x) {
            const int e = v.bpaths[x];
            if (!(e & 1)) atomicAdd(&own, 1);
            const bool path = e >= 0 && (e >> 1) < v.P;
            const int c = !path ? -1 : (e & 1) ? v.bdi[e >> 1] : v.bci[e >> 1];
            if (c < t0 || c >= t1 || x < v.bptr[c] || x >= v.bptr[c + 1]) bad = 1;
        }
    for (long l = (long)blockIdx.x * blockDim.x + threadIdx.x; l < v.NLV; l += (long)gridDim.x * blockDim.x) {
        const int c = v.lci[l];
        if (c < 0 || c >= v.N || (l > 0 && v.lci[l - 1] >= c) || !(v.flags[c] & CMF_CELL_LEVEE)) bad = 1;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    int* most = v.ctl + kCtlTileMax;
    if (v.features & CMF_FEAT_BIFURCATION) atomicMax(most, v.bptr[t1] - v.bptr[t0]);
    atomicMax(most + 1, own);
    int listed = 0;
    if (v.NLV > 0) listed = first_at_least(v.lci, (int)v.NLV, t1) - first_at_least(v.lci, (int)v.NLV, t0);
    atomicMax(most + 2, listed);
    atomicMax(most + 3, dams);
    if (hi > 0) atomicMax(most + 4, hi - lo);
    if (bad || levees != listed || (hi > 0 && beyond != hi - lo)) atomicMax(most + 5, 1);
    atomicMax(most + 6, cell_ends);
    atomicAdd(most + 7, stray);
}

template <typename REAL, bool RES, bool LEV, bool BIF>
__global__ void __launch_bounds__(resident_threads<REAL>(), 1)
k_resident(const Dev<REAL> v, const StatsArgs stats, const ResidentArgs a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int quit, step_max, own_paths, own_dams, levee_range[2], halo_lo, halo_hi, taken[2];
    const Tile<REAL> t = tile_of(v, a, smem);
    const int tid = threadIdx.x, nthr = blockDim.x;
    Wait w{v.ctl, v.status, &quit, (unsigned)v.ctl[kCtlEpoch], a.polls};

    // ---- load the tile ----
    if (tid == 0) {
        quit = own_paths = own_dams = halo_hi = taken[0] = taken[1] = 0;
        step_max = 1;
        halo_lo = INT32_MAX;
    }
    if (LEV && tid < 2) levee_range[tid] = first_at_least(v.lci, (int)v.NLV, t.t0 + (tid ? t.count : 0));
    __syncthreads();
    const REAL T = v.outer[0];
    int n_steps = 1;
    const int ends0 = BIF ? v.bptr[t.t0] : 0;
    for (int j = tid; j < t.count; j += nthr) {
        const int i = t.t0 + j;
        uint8_t fl = v.flags[i] & ~(kRemoteDown | kRemoteUp);  // no CMF_CELL_* bits: a caller may use them
        const int dn = v.dn[i], c0 = v.up[i], c1 = upstream_end(v, (long)i);
        t.dn[j] = dn;
        t.c0[j] = c0;
        t.c1[j] = c1;
        if (!t.has(dn)) fl |= kRemoteDown;
        if (c0 < c1 && !(t.has(c0) && t.has(c1 - 1))) {
            fl |= kRemoteUp;
            atomicMin(&halo_lo, max(c0, t.t0 + t.count));
            atomicMax(&halo_hi, c1);
        }
        t.fl[j] = fl;
        t.rs[j] = v.rs0[i];
        t.fs[j] = v.fs0[i];
        t.at(RF_WIDTH, j) = v.rw[i];
        t.at(RF_LEN, j) = v.rl[i];
        t.at(RF_BANK, j) = v.rh[i];
        t.at(RF_NRIV, j) = v.rman[i];
        t.at(RF_NFLD, j) = v.fman[i];
        t.at(RF_ELEV, j) = v.celv[i];
        t.at(RF_DX, j) = v.dnd[i];
        t.at(RF_AREA, j) = v.ca[i];
        t.at(RF_RUNOFF, j) = v.runoff[i];
        t.at(RF_ROUT, j) = v.rout[i];
        t.at(RF_FOUT, j) = v.fout[i];
        t.at(RF_RDEP, j) = v.rdep[i];
        t.at(RF_FDEP, j) = v.fdep[i];
        t.at(RF_RCSD, j) = v.rcsd[i];
        t.at(RF_FCSD, j) = v.fcsd[i];
        t.at(RF_FCSA, j) = v.fcsa[i];
        if (a.o_rows) {
            REAL* rows = reinterpret_cast<REAL*>(smem + a.o_rows);
            for (int l = 0; l < v.K; ++l) rows[l * t.stride + j] = v.tbl[(long)i * v.K + l];
        }
        if (BIF) {
            t.end_of[j] = v.bptr[i] - ends0;
            if (j == t.count - 1) t.end_of[j + 1] = v.bptr[i + 1] - ends0;
            for (int b = v.bptr[i]; b < v.bptr[i + 1]; ++b) {
                const int e = v.bpaths[b], p = e >> 1, x = b - ends0;
                const int other = (e & 1) ? v.bci[p] : v.bdi[p];
                t.end[x] = e;
                t.end_other[x] = t.has(other) ? other - t.t0 : -1;
                if (!(e & 1)) {
                    const int s = atomicAdd(&own_paths, 1);
                    t.path[s] = p;
                    t.path_a[s] = j;
                    t.path_b[s] = t.end_other[x];
                    t.path_xa[s] = x;
                    t.path_xb[s] = -1;
                    t.plen[s] = v.blen[p];
                }
            }
        }
        if (RES && (fl & CMF_CELL_RESERVOIR)) {
            const int s = atomicAdd(&own_dams, 1);
            const DamRule<REAL> r = dam_rule_of(v, i);
            t.dam_of[j] = (uint16_t)s;
            t.rti[s] = v.rti[i];
            t.dam_at(DF_CONS, s) = r.v_cons;
            t.dam_at(DF_ADJ, s) = r.v_adj;
            t.dam_at(DF_EMERG, s) = r.v_emerg;
            t.dam_at(DF_NORM, s) = r.q_norm;
            t.dam_at(DF_QADJ, s) = r.q_adj;
            t.dam_at(DF_FLOOD, s) = r.q_flood;
        }
        if (a.fixed_n <= 0 && !(RES && (fl & CMF_CELL_DAM_RELATED)))
            n_steps = max(n_steps, cfl_steps<REAL>(t.at(RF_DX, j), t.at(RF_RDEP, j), v.cfl_alpha, v.g, v.max_dt, T));
    }
    const int levees = LEV ? levee_range[1] - levee_range[0] : 0, levee0 = LEV ? levee_range[0] : 0;
    for (int s = tid; s < levees; s += nthr) {
        const long li = levee0 + s;
        const int i = v.lci[li], j = i - t.t0;
        t.levee_cell[s] = j;
        t.levee_of[j] = (uint16_t)s;
        t.ps[s] = v.ps[i];
        t.levee_at(LF_PDEP, s) = v.pdep[i];
        t.levee_at(LF_CROWN, s) = v.lcrown[li];
        t.levee_at(LF_FRAC, s) = v.lfrac[li];
        t.levee_at(LF_BASE, s) = v.lbase[li];
        for (int f = 0; f < 6; ++f) t.levee_at(LF_SBASE + f, s) = v.lmk[f * v.NLV + li];
    }
    __syncthreads();
    const int paths = BIF ? own_paths : 0;
    const int ends = BIF ? t.end_of[t.count] : 0;
    const int halo0 = halo_lo, halo = halo_hi > 0 ? halo_hi - halo_lo : 0;
    if (BIF) {
        // the own paths' levels; and the second ends of own paths find them
        for (int x = tid; x < paths * v.L; x += nthr) {
            const int s = x / v.L, l = x - s * v.L;
            const TilePathLevels<REAL> lv{t, s, v.L};
            const long g = (long)t.path[s] * v.L + l;
            lv.at(PL_SILL, l) = v.belv[g];
            lv.at(PL_WIDTH, l) = v.bwid[g];
            lv.at(PL_NRIV, l) = v.bman[g];
            lv.at(PL_FLUX, l) = v.bout[g];
            lv.at(PL_DEPTH, l) = v.bcsd[g];
        }
        for (int s = tid; s < paths; s += nthr) {
            const int jb = t.path_b[s];
            if (jb < 0) continue;
            for (int b = t.end_of[jb]; b < t.end_of[jb + 1]; ++b)
                if (t.end[b] == 2 * t.path[s] + 1) t.path_xb[s] = b;
        }
    }

    // ---- sub-step count: the maximum over all tiles ----
    int n = a.fixed_n;
    if (n <= 0) {
        n_steps = __reduce_max_sync(0xffffffffu, n_steps);
        if ((tid & 31) == 0) atomicMax(&step_max, n_steps);
        __syncthreads();
        if (tid == 0) atomicMax(&v.ctl[kCtlCflMax], step_max);
    }
    if (tiles_meet(v.rflag, v.ctl, v.status, (int)gridDim.x, a.polls, &quit)) return;
    if (n <= 0) n = __ldcg(v.ctl + kCtlCflMax);
    if (n < 1) n = 1;
    const int cap = v.max_sub_cap > 0 ? v.max_sub_cap : kHardSubStepCap;
    if (n > cap) {
        if (tid == 0) atomicOr(v.status, CMF_STATUS_SUBSTEP_CAP);
        n = cap;
    }
    const REAL dt = (REAL)(v.tsec[0] / (double)n);
    // The epochs of this interval are taken from here on, by every tile that gets
    // here: all have read the last one, and an interval that is given up leaves
    // words with them, which the next one must not take for its own.
    if (tid == 0) v.ctl[kCtlEpoch] = (int)(w.epoch + 1 + n);
    w.epoch += 1;
    for (int j = tid; j < t.count; j += nthr) publish_state<REAL, RES, LEV, BIF>(v, t, j, w.epoch);

    // The warps take the paths in chunks of 32 / kPathLanes and the cells in
    // chunks of 32, the first chunks by warp index and the rest as they come
    // free: a tile has one to two chunks per warp, and their lengths differ.
    // The paths, whose chain is the longest, go to the last warps, because the
    // first ones fetch the other tiles' values next.
    constexpr int kPathsPerWarp = 32 / kPathLanes;
    const int warp = tid >> 5, lane = tid & 31, warps = nthr >> 5;
    const int cell_chunks = (t.count + 31) / 32, path_chunks = (paths + kPathsPerWarp - 1) / kPathsPerWarp;
    const int chunks = cell_chunks + path_chunks;
    auto next_chunk = [&](int* taken) {
        if (chunks <= warps) return chunks;
        int c = 0;
        if (lane == 0) c = atomicAdd(taken, 1);
        return warps + __shfl_sync(0xffffffffu, c, 0);
    };
    for (int k = 0; k < n; ++k, ++w.epoch) {
        if (k == a.leave_step && blockIdx.x == gridDim.x - 1) return;
        const bool diag = k == n - 1;
        const bool want_fraction = diag || stats.count > 0;
        for (int c = warps - 1 - warp; c < chunks; c = next_chunk(&taken[0])) {
            if (BIF && c < path_chunks) {
                const int s = c * kPathsPerWarp + lane / kPathLanes, level = lane % kPathLanes;
                resident_path_momentum<REAL, RES, LEV>(v, t, w, min(s, paths - 1), level, s < paths && level < v.L, dt);
            } else {
                const int j = (c - path_chunks) * 32 + lane;
                if (j < t.count) resident_momentum<REAL, RES, LEV>(v, t, w, j, dt, diag);
                __syncwarp();
            }
        }
        if (tid == 0) taken[1] = 0;
        if (halo + ends > 0) fetch_fluxes<REAL, BIF>(v, t, w, halo0, halo, ends);
        __syncthreads();
        for (int j = tid; j < t.count; j += nthr) resident_limit<REAL, BIF>(v, t, w, j, dt, halo0);
        if (halo + ends > 0) fetch_rates<REAL, BIF>(v, t, w, halo0, halo, ends);
        __syncthreads();
        for (int c = warp; c < chunks; c = next_chunk(&taken[1])) {
            if (c < cell_chunks) {
                const int j = c * 32 + lane;
                if (j < t.count) resident_stage<REAL, RES, LEV, BIF>(v, t, w, j, dt, halo0, diag, want_fraction);
                __syncwarp();
            } else if (BIF) {
                const int s = (c - cell_chunks) * kPathsPerWarp + lane / kPathLanes, level = lane % kPathLanes;
                if (s < paths && level < v.L) {
                    const int b = t.path_b[s];
                    const REAL lr_c = t.at(RF_LR, t.path_a[s]);
                    const REAL lr_d = b >= 0 ? t.at(RF_LR, b) : t.end_at(PE_RATE, t.path_xa[s]);
                    REAL& o = TilePathLevels<REAL>{t, s, v.L}.at(PL_FLUX, level);
                    o = (o >= (REAL)0) ? o * lr_c : o * lr_d;
                }
                __syncwarp();
            }
        }
        if (tid == 0) taken[0] = 0;
        if (LEV) {
            __syncthreads();
            for (int s = tid; s < levees; s += nthr)
                resident_levee<REAL, RES, LEV, BIF>(v, t, s, levee0, w.epoch + 1, diag, want_fraction);
        }
        if (cta_quits(&quit)) return;
        if (stats.count > 0) {
            if (stats.need_weight && t.t0 == 0 && tid == 0)
                stats.weight[0] = __dadd_rn(stats.weight[0], (double)dt);
            for (int j = tid; j < t.count; j += nthr) {
#pragma unroll 1
                for (int q = 0; q < stats.count; ++q) {
                    if (stats.op[q] == CMF_STAT_LAST) continue;
                    fold_stat(stats.out[q] + t.t0 + j, stats.op[q], resident_stat(v, t, stats.var[q], j), (double)dt);
                }
            }
        }
    }

    // ---- write the state back ----
    for (int j = tid; j < t.count; j += nthr) {
        const int i = t.t0 + j;
        v.rs0[i] = t.rs[j];
        v.fs0[i] = t.fs[j];
        v.rout[i] = t.at(RF_ROUT, j);
        v.fout[i] = t.at(RF_FOUT, j);
        v.rdep[i] = t.at(RF_RDEP, j);
        v.fdep[i] = t.at(RF_FDEP, j);
        v.rcsd[i] = t.at(RF_RCSD, j);
        v.fcsd[i] = t.at(RF_FCSD, j);
        v.fcsa[i] = t.at(RF_FCSA, j);
    }
    for (int j = tid; RES && j < t.count; j += nthr)
        if (t.fl[j] & CMF_CELL_RESERVOIR) v.rti[t.t0 + j] = t.rti[t.dam_of[j]];
    for (int s = tid; s < levees; s += nthr) {
        const int i = t.t0 + t.levee_cell[s];
        v.ps[i] = t.ps[s];
        v.pdep[i] = t.levee_at(LF_PDEP, s);
    }
    for (int x = tid; x < paths * v.L; x += nthr) {
        const int s = x / v.L, l = x - s * v.L;
        const TilePathLevels<REAL> lv{t, s, v.L};
        const long g = (long)t.path[s] * v.L + l;
        v.bout[g] = lv.at(PL_FLUX, l);
        v.bcsd[g] = lv.at(PL_DEPTH, l);
    }
    if (blockIdx.x == 0 && tid == 0) {
        v.dt[0] = dt;
        v.nsub[0] = n;
        v.cur[0] = n - 1;
        v.ctl[kCtlMaxSteps] = n;
        v.ctl[kCtlStep] = n;
    }
}

}  // namespace cmf

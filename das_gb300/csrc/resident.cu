// resident.cu -- the acoustic time loop with its wavefields kept on chip.
//
// A shot's grid is cut into gx x gz tiles, one per CTA and one CTA per SM, and ONE
// cooperative launch advances it by many steps.  For the whole launch a CTA keeps its
// tile in the SM: p_curr and p_prev in shared memory (p_next overwrites p_prev in place:
// a cell's p_prev is read only by the thread that computes its p_next), vel^2 dt^2 and
// the illumination or image accumulator in tensor memory, each thread its own words.
// Off the chip go only the two outermost rows and columns of every tile, once per step,
// and what a shot keeps: snapshots, traces, and the state at the end of the launch.
//
// Why: one launch per step reloads every operand (16 bytes a point) from L2 or HBM and
// pays the fixed chain of a launch, about 6 us, each step.  Here a step costs its
// arithmetic, and the exchange of a tile's edge hides behind the tile's interior.
// Measured on GB300, us per step, one launch per step -> here: 150 x 400 5.6 -> 1.5
// forward, 6.2 -> 1.8 in a migration; 301 x 1203 5.8 -> 1.75, 6.5 -> 2.1; 600 x 2000 6.9 ->
// 2.7, 7.6 -> 3.3; 1000 x 4000 11.2 -> 5.2, 13.4 -> 6.7 (600 Gpts/s).  Small grids are
// bound by the chain edge -> packet -> neighbour's halo (about 1.4 us), large ones by
// issue slots: some 110 instructions per four points, half of the slots used.  The
// arithmetic is packed (.f32x2) for those slots; a packed instruction takes the pipe as
// long as the two it replaces.
//
// Work inside a CTA (15 compute warps, one halo warp).  A unit is four points of one row.
//   * Phase E: the tile's edge units (first and last column, two first and two last
//     rows), one per thread.  They are computed first and published to the neighbours
//     at once, so that the exchange runs while
//   * phase I computes the other units: a thread owns one column of units over up to
//     RS_MAXR consecutive rows, with a five-row register window along z.  (The x
//     neighbours come from shared memory: as register pairs, ready for the packed
//     arithmetic; from the adjacent lanes, by shuffles and selects, they cost ten more
//     instructions of a hundred.)
//   * The halo warp collects the neighbours' edges meanwhile into the halo of p_next,
//     samples the receivers of the last step, stages the next one's injection values from
//     registers it loaded a step before, and prefetches the next snapshot into L2.  (It runs
//     a loop of its own: what it keeps from step to step costs the compute warps nothing.)
// One barrier ends the step.
//
// Exchange: 16-byte packets {value, tag, value, tag} in global memory, tag = step
// number; each 8-byte half is written and read whole, so a matching tag vouches for the
// value beside it and no fence or flag round trip is needed (measured 0.73 us from one
// CTA's store to the next step of its neighbour).  Two slots per tile, by step parity:
// a tile writes step k+2's packet only after it has received its neighbour's step k+1,
// which that neighbour sent after it had read step k's.  Every wait is bounded; all CTAs
// are resident at once (cooperative launch).
//
// Arithmetic: the reference's operation order with every operation rounded (no
// contraction), as in acoustic_kernels.cuh, so finite results are bit-identical to it but for
// the sign of a zero (2c - p_prev is formed as -(p_prev - 2c), see rs_stencil).
// Cells the reference never writes stay zero unless receivers inject into them: the
// source and the receivers' row must lie on interior rows (rs_shot_fits), so the only
// such cells are the four of that row beside the left and right edges.  Their values in
// the reference's three rotating buffers are kept in a small ring (quirk Q1).
#include "resident.cuh"

namespace w2d {

// ---- device: packed pairs ----------------------------------------------------------
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f32x2 v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// A packed product that stays one: a multiply followed by an add becomes a fused
// multiply-add in the assembler even with explicit rounding, so the product is formed as
// a*b + z with z = -0 read from memory (adding -0 changes no value, and the assembler
// cannot know it).  Both forms occupy the pipe alike.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 z)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(z));
    return r;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// four points of a row as two pairs
struct F4 {
    f32x2 a, b;
};
__device__ __forceinline__ F4 ld_f4(const float* p)
{
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return F4{v.x, v.y};
}
__device__ __forceinline__ void st_f4(float* p, const F4& v)
{
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.a, v.b);
}
__device__ __forceinline__ void f4_get(const F4& v, float u[4])
{
    upk(v.a, u[0], u[1]);
    upk(v.b, u[2], u[3]);
}
__device__ __forceinline__ F4 f4_neg(const F4& v)
{
    const f32x2 sign = 0x8000000080000000ull;
    return F4{v.a ^ sign, v.b ^ sign};
}
__device__ __forceinline__ F4 f4_of(const float u[4]) { return F4{pk(u[0], u[1]), pk(u[2], u[3])}; }

// ---- device: tensor memory as each thread's own words --------------------------------
__device__ __forceinline__ void tm_ld4(uint32_t addr, uint32_t r[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// the registers of the loads in flight pass through the wait: no use moves above it
__device__ __forceinline__ void tm_wait_ld(uint32_t r[4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]));
}
__device__ __forceinline__ void tm_wait_ld2(uint32_t r[4], uint32_t s[4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(s[0]), "+r"(s[1]),
                   "+r"(s[2]), "+r"(s[3]));
}
__device__ __forceinline__ void tm_st4(uint32_t addr, const uint32_t r[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]));
}
__device__ __forceinline__ void tm_wait_st()
{
    asm volatile("tcgen05.wait::st.sync.aligned;");
}
// The tensor-memory instructions are the whole warp's: its lanes meet first.  (Not
// __syncwarp, which would also keep shared-memory loads from moving ahead of it.)
__device__ __forceinline__ void tm_converge() { asm volatile("bar.warp.sync 0xffffffff;"); }
__device__ __forceinline__ F4 f4_bits(const uint32_t r[4])
{
    return F4{pk(__uint_as_float(r[0]), __uint_as_float(r[1])),
              pk(__uint_as_float(r[2]), __uint_as_float(r[3]))};
}
__device__ __forceinline__ void bits_f4(const F4& v, uint32_t r[4])
{
    float u[4];
    f4_get(v, u);
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = __float_as_uint(u[j]);
}
__device__ __forceinline__ void bits_of(const float4& v, uint32_t r[4])
{
    r[0] = __float_as_uint(v.x);
    r[1] = __float_as_uint(v.y);
    r[2] = __float_as_uint(v.z);
    r[3] = __float_as_uint(v.w);
}

// words of one thread: model rows, edge unit's model, accumulator rows, edge accumulator
constexpr int RS_TM_C = 0, RS_TM_CE = 60, RS_TM_A = 64, RS_TM_AE = 124;

// ---- device: packets ---------------------------------------------------------------
struct RsPacket {
    unsigned long long a, b;
};
__device__ __forceinline__ void rs_send(uint4* p, float a, float b, unsigned tag)
{
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p),
                 "l"(t | __float_as_uint(a)), "l"(t | __float_as_uint(b))
                 : "memory");
}
// (relaxed, not volatile: volatile loads wait for one another)
__device__ __forceinline__ RsPacket rs_peek(const uint4* p)
{
    RsPacket v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p));
    return v;
}

// One step of four points: reference operation order, every operation rounded.
// l, r: the two points left and right of c; w0, w1, w3, w4: rows z-2..z+2.
struct RsConst {
    f32x2 k0, k1, k2, dx2, dz2, m2, z;
};
__device__ __forceinline__ F4 rs_stencil(const RsConst& k, const F4& w0, const F4& w1, const F4& c,
                                         const F4& w3, const F4& w4, f32x2 l, f32x2 r,
                                         const F4& pp, const F4& v, F4& lap)
{
    float cx, cy, cz, cw, l2, l1, r1, r2;
    upk(l, l2, l1);
    upk(r, r1, r2);
    upk(c.a, cx, cy);
    upk(c.b, cz, cw);
    auto mul = [&](f32x2 a, f32x2 b) { return mul2(a, b, k.z); };
    const f32x2 kca = mul(k.k0, c.a), kcb = mul(k.k0, c.b);
    // (c2*(m2+p2) + c1*(m1+p1)) + c0*c along x, then along z
    const f32x2 xa = mul(add2(add2(mul(k.k2, add2(l, c.b)),
                                   mul(k.k1, pk(fadd(l1, cy), fadd(cx, cz)))), kca), k.dx2);
    const f32x2 xb = mul(add2(add2(mul(k.k2, add2(c.a, r)),
                                   mul(k.k1, pk(fadd(cy, cw), fadd(cz, r1)))), kcb), k.dx2);
    const f32x2 za = mul(add2(add2(mul(k.k2, add2(w0.a, w4.a)), mul(k.k1, add2(w1.a, w3.a))),
                              kca), k.dz2);
    const f32x2 zb = mul(add2(add2(mul(k.k2, add2(w0.b, w4.b)), mul(k.k1, add2(w1.b, w3.b))),
                              kcb), k.dz2);
    // v*lap + (2c - pp), the second term as -(pp - 2c): 2c is exact, so one rounding.  (Where
    // 2c overflows the Laplacian has: the cell is infinite or NaN in either form.)
    lap.a = add2(xa, za);
    lap.b = add2(xb, zb);
    F4 u;
    u.a = sub2(mul(v.a, lap.a), fma2(c.a, k.m2, pp.a));
    u.b = sub2(mul(v.b, lap.b), fma2(c.b, k.m2, pp.b));
    return u;
}

// A CTA's tile, at the start of its dynamic shared memory; the arrays as float offsets
// from there, so that every access is a shared-memory access also in functions of their own.
struct RsTile {
    int nx, nz, ldx, fs;
    int x0, z0, ncol, nrows, pitch;  // pitch: floats of a shared-memory row
    int left, right;                 // whether there are neighbours
    int rec_row, src_row, src_x;     // local row, and column of the source (-1: not here)
    int mirror;                      // local row of z = 2 under a free surface, -1: not here
    int plane[2];                    // p_curr / p_prev: two halo rows, the tile's, two more
    int hx;                          // float2 [parity][side][row]: columns beside the tile
    int inj;                         // [parity][pitch]: added to the receiver row
    int injs;                        // [parity]: added to the source cell
    int pre;                         // [parity]: the source cell before that
    int ring;                        // [3][4]: never-written cells of the receiver row
    int fx, fz;                      // sponge by column, by row
    int rk;                          // receiver of a column, -1: none
    int n_l, n_lr, n_lrt, n_in;      // packets of a step: from the left, and the right, and
                                     // above, and below
    int half, in;                    // packets of one slot; where this tile's begin
    int nci, nseg, R;                // phase I: columns, segments, rows of a segment
    int tm;                          // tensor-memory address
    int next;                        // [parity]: groups of packets taken
    float dx2, dz2;
    float z;                         // -0
};
static_assert(sizeof(RsTile) <= RS_TILE_FLOATS * 4 && sizeof(RsShot) <= RS_SHOT_FLOATS * 4 &&
                  sizeof(RsShot) % 4 == 0,
              "the tile's and the shot's records fit their places");

constexpr int RS_PLANE0 = RS_TILE_FLOATS + RS_SHOT_FLOATS;  // where the first plane begins

extern __shared__ __align__(128) float rs_smem[];
__device__ __forceinline__ const RsTile& rs_tile() { return *reinterpret_cast<RsTile*>(rs_smem); }
__device__ __forceinline__ f32x2 rs_pair(int o) { return *reinterpret_cast<f32x2*>(rs_smem + o); }

// Which of the four never-written cells of a row column ix is.
__device__ __forceinline__ int rs_cell(int ix, int nx) { return ix < 2 ? ix : 4 + ix - nx; }

// The rules of the receiver row, the source row and the free surface for the unit at
// column c of a row, whose new values are u (zero on never-written columns: those not in
// xm).  par: parity of the step; nb: which of the three rotating buffers p_next is.
// (Receivers are sampled by the halo warp, from p_curr of the next step: this is on the
// way from a tile's edge to its neighbours.)
__device__ __forceinline__ F4 rs_special(const F4& v, int nxt, int row, int c, int par, int nb,
                                         unsigned xm, int pitch, bool inject)
{
    const RsTile& t = rs_tile();
    const int rec_row = t.rec_row, src_row = t.src_row, mirror = t.mirror, inj = t.inj;
    float u[4];
    f4_get(v, u);
    const bool at_rec = row == rec_row && inject;
    float* ring = rs_smem + t.ring + 4 * nb;
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (at_rec) d = *reinterpret_cast<const float4*>(rs_smem + inj + par * pitch + 4 * c);
    const int ix = t.x0 + 4 * c;
    if (row == rec_row && xm != 15u) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (!((xm >> j) & 1u) && ix + j < t.nx) u[j] = ring[rs_cell(ix + j, t.nx)];
    }
    if (row == mirror)  // p_next[1,:] = -p_next[2,:] over every column
        *reinterpret_cast<float4*>(rs_smem + nxt + (row + 1) * pitch + 4 * c) =
            make_float4(-u[0], -u[1], -u[2], -u[3]);
    if (at_rec) {
        u[0] = fadd(u[0], d.x);
        u[1] = fadd(u[1], d.y);
        u[2] = fadd(u[2], d.z);
        u[3] = fadd(u[3], d.w);
        if (xm != 15u) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (!((xm >> j) & 1u) && ix + j < t.nx) ring[rs_cell(ix + j, t.nx)] = u[j];
        }
    }
    if (row == src_row && c == t.src_x >> 2) {
        const float w = rs_smem[t.injs + par];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j == (t.src_x & 3)) {
                rs_smem[t.pre + par] = u[j];
                u[j] = fadd(u[j], w);
            }
    }
    return f4_of(u);
}

// Receiver samples of the step whose p_next is now the plane at pl: row[r] for every
// receiver r of the tile (the whole warp).  par: parity of that step.
__device__ __forceinline__ void rs_sample(float* row, int pl, int par)
{
    const RsTile& t = rs_tile();
    const int src_x = t.src_row == t.rec_row ? t.src_x : -1, ncol = t.ncol;
    const float* at = rs_smem + pl + (t.rec_row + 2) * t.pitch;
    const float* rk = rs_smem + t.rk;
    const float before = rs_smem[t.pre + par];  // without the next step's injection
#pragma unroll 2
    for (int c = threadIdx.x & 31; c < ncol; c += 32) {  // a unit a lane
        const int4 r = *reinterpret_cast<const int4*>(rk + 4 * c);
        float4 v = *reinterpret_cast<const float4*>(at + 4 * c);
        if (src_x >> 2 == c) {
            if ((src_x & 3) == 0) v.x = before;
            if ((src_x & 3) == 1) v.y = before;
            if ((src_x & 3) == 2) v.z = before;
            if ((src_x & 3) == 3) v.w = before;
        }
        if (r.x >= 0) row[r.x] = v.x;
        if (r.y >= 0) row[r.y] = v.y;
        if (r.z >= 0) row[r.z] = v.z;
        if (r.w >= 0) row[r.w] = v.w;
    }
}

// Pointwise work of a fused step on one unit of p_curr: snapshot copy and illumination
// (forward), or imaging with the forward snapshot f (backward).
__device__ __forceinline__ F4 rs_illum(const F4& acc, const F4& c, f32x2 z)
{
    return F4{add2(acc.a, mul2(c.a, c.a, z)), add2(acc.b, mul2(c.b, c.b, z))};
}
__device__ __forceinline__ F4 rs_image(const F4& acc, const F4& c, const float4& f, f32x2 dt,
                                       f32x2 z)
{
    return F4{add2(acc.a, mul2(mul2(pk(f.x, f.y), c.a, z), dt, z)),
              add2(acc.b, mul2(mul2(pk(f.z, f.w), c.b, z), dt, z))};
}
__device__ __forceinline__ void rs_snap(float* dst, const F4& c)
{
    float u[4];
    f4_get(c, u);
    __stcs(reinterpret_cast<float4*>(dst), make_float4(u[0], u[1], u[2], u[3]));
}
// u times the sponge, and zero on never-written columns (xm: bit j, column j interior)
__device__ __forceinline__ F4 rs_frame(const F4& u, const float4& fx, float fz, unsigned xm,
                                       f32x2 z)
{
    F4 v{mul2(u.a, pk(fminf(fx.x, fz), fminf(fx.y, fz)), z),
         mul2(u.b, pk(fminf(fx.z, fz), fminf(fx.w, fz)), z)};
    if (xm != 15u) {
        float s[4];
        f4_get(v, s);
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = (xm >> j) & 1u ? s[j] : 0.0f;
        v = f4_of(s);
    }
    return v;
}

// A thread's units.  Only what a step needs of them stays in registers (there are no
// more than 128 a thread, and local memory would go to L2: the shared memory of a CTA
// leaves next to no L1): the rest is read from the tile's record.
struct RsMine {
    // edge unit: row, unit column << 16, and whether there is one (bit 31), it is written
    // (bit 30), a rule of its own applies (bit 29), it is the last column's (bit 28); packets it
    // sends along x and z, as indices into the packet buffer, -1: none
    unsigned e;
    int ox, oz;
    // interior units: unit column, first row << 8, number of rows << 24 (0: none)
    unsigned i;
    // rows (bit j: the j-th) with a rule of their own; above, the interior columns of the
    // edge unit (bits 16-19) and of the interior units (bits 20-23), and whether the warp's
    // interior units (bit 24) or edge units (bit 25) meet the sponge or the edge columns
    unsigned b;
    unsigned h;           // edge column: its cells beside the tile in RsTile::hx, and (above
                          // bit 16) how far the other parity's are
    uint32_t tm;          // tensor-memory address of this thread's words

    __device__ __forceinline__ int er() const { return e & 0xffff; }
    __device__ __forceinline__ int ec() const { return (e >> 16) & 0xff; }
    __device__ __forceinline__ bool e_live() const { return e >> 31; }
    __device__ __forceinline__ bool e_write() const { return (e >> 30) & 1u; }
    __device__ __forceinline__ bool e_spec() const { return (e >> 29) & 1u; }
    __device__ __forceinline__ bool last_col() const { return (e >> 28) & 1u; }
    __device__ __forceinline__ int c() const { return i & 0xff; }
    __device__ __forceinline__ int r0() const { return (i >> 8) & 0xffff; }
    __device__ __forceinline__ int n() const { return i >> 24; }
    __device__ __forceinline__ unsigned spec() const { return b & 0x7fffu; }
    __device__ __forceinline__ unsigned e_xm() const { return (b >> 16) & 15u; }
    __device__ __forceinline__ unsigned i_xm() const { return (b >> 20) & 15u; }
    __device__ __forceinline__ bool i_frame() const { return (b >> 24) & 1u; }
    __device__ __forceinline__ bool e_frame() const { return (b >> 25) & 1u; }
    __device__ __forceinline__ int hx(int par) const
    {
        return (int)(h & 0xffffu) + (par ? (int)(h >> 16) : 0);
    }
};
static_assert(RS_MAXR <= 15, "rows with a rule: 15 bits");

// What this step does beside the stencil.
struct RsFused {
    float* snap_out;         // forward: copy of p_curr, or (lap) its Laplacian
    const float* snap_in;    // backward: the forward snapshot to image with
    bool acc;                // illumination or image
    bool lap;
    bool fold;               // adjoint under a free surface: the first row is z = 2
};

// Phase I of one step: rows of one unit column.  FUSED: see RsFused.
template <bool FUSED>
__device__ __forceinline__ void rs_inner(const RsMine& m, const RsConst& k, int pitch, int cur,
                                         int nxt, int R, const RsFused& fu, f32x2 img_dt)
{
    const RsTile& t = rs_tile();
    const bool frame = m.i_frame();
    const int c = m.c(), r0 = m.r0(), n = m.n();
    // addresses advance by rows and stay on the thread's last one
    int oc = cur + (r0 + 2) * pitch + 4 * c;
    const int dn = nxt - cur;
    F4 w0 = ld_f4(rs_smem + oc - 2 * pitch), w1 = ld_f4(rs_smem + oc - pitch),
       w2 = ld_f4(rs_smem + oc), w3 = ld_f4(rs_smem + oc + pitch);
    float4 fx = make_float4(1.f, 1.f, 1.f, 1.f);
    if (frame) fx = *reinterpret_cast<const float4*>(rs_smem + t.fx + 4 * c);
    const int ofz = frame ? t.fz + r0 : 0;
    uint32_t cb[4], ab[4];
    tm_ld4(m.tm + RS_TM_C, cb);
    size_t goff = 0;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f), f1 = f;  // two rows of the snapshot ahead
    if (FUSED) {
        if (fu.acc) tm_ld4(m.tm + RS_TM_A, ab);
        goff = (size_t)(t.z0 + r0) * t.ldx + t.x0 + 4 * c;
        if (fu.snap_in && n) f = __ldcs(reinterpret_cast<const float4*>(fu.snap_in + goff));
        if (fu.snap_in && n > 1)
            f1 = __ldcs(reinterpret_cast<const float4*>(fu.snap_in + goff + t.ldx));
    }
#pragma unroll 5
    for (int i = 0; i < R; ++i) {
        const bool ok = i < n;
        tm_converge();
        if (FUSED && fu.acc) tm_wait_ld2(cb, ab);
        else tm_wait_ld(cb);
        const F4 v = f4_bits(cb);
        F4 acc{0, 0};
        if (FUSED && fu.acc) acc = f4_bits(ab);
        if (i + 1 < R) {
            tm_ld4(m.tm + RS_TM_C + 4 * (i + 1), cb);
            if (FUSED && fu.acc) tm_ld4(m.tm + RS_TM_A + 4 * (i + 1), ab);
        }
        float4 f2 = f1;
        if (FUSED && fu.snap_in && i + 2 < n)
            f2 = __ldcs(reinterpret_cast<const float4*>(fu.snap_in + goff + 2 * (size_t)t.ldx));
        const F4 w4 = ld_f4(rs_smem + oc + 2 * pitch);
        const F4 pp = ld_f4(rs_smem + oc + dn);
        const f32x2 l = rs_pair(oc - 2), r = rs_pair(oc + 4);
        if (FUSED && i == 0 && fu.fold) {
            w1 = f4_neg(w2);
            w0 = f4_neg(w3);
        }
        F4 lap;
        F4 u = rs_stencil(k, w0, w1, w2, w3, w4, l, r, pp, v, lap);
        if (FUSED && i == 0 && fu.fold) w1 = F4{0, 0};
        if (frame) u = rs_frame(u, fx, rs_smem[ofz + (ok ? i : 0)], m.i_xm(), k.z);
        if (ok) st_f4(rs_smem + oc + dn, u);
        if (FUSED) {
            if (fu.acc) {
                acc = fu.snap_in ? rs_image(acc, w2, f, img_dt, k.z) : rs_illum(acc, w2, k.z);
                uint32_t o[4];
                bits_f4(acc, o);
                tm_converge();
                tm_st4(m.tm + RS_TM_A + 4 * i, o);
            }
            if (fu.snap_out && ok) rs_snap(fu.snap_out + goff, fu.lap ? lap : w2);
            f = f1;
            f1 = f2;
            goff += t.ldx;
        }
        if (i + 1 < n) oc += pitch;
        w0 = w1;
        w1 = w2;
        w2 = w3;
        w3 = w4;
    }
    if (FUSED && fu.acc) tm_wait_st();
}

// This step's packets (at src) into the halo of p_next, FLIGHT groups of 32 at a time: the
// halo warp from the start of the step, and every compute warp that is done with its units
// takes its share of what is left (next: the step's counter of groups taken).  False: a
// wait gave up (recorded), or another CTA's did.  (Looking at a sample of the packets
// before all of them are looked at measured slower: one more round trip, 2.0 -> 2.3 us a
// step at 150 x 400, 7.7 -> 8.3 at 1000 x 4000.)
template <int FLIGHT>
__device__ __forceinline__ bool rs_collect(const uint4* src, unsigned tag, int nxt, int par,
                                           int next, unsigned* err)
{
    const RsTile& t = rs_tile();
    const int n_in = t.n_in, lane = threadIdx.x & 31;
    for (;;) {
        int g = 0;
        if (lane == 0) g = atomicAdd(reinterpret_cast<int*>(rs_smem + next), FLIGHT);
        const int b0 = 32 * __shfl_sync(0xffffffffu, g, 0) + lane;
        if (b0 - lane >= n_in) return true;
        unsigned left = 0;
#pragma unroll
        for (int j = 0; j < FLIGHT; ++j) left |= b0 + 32 * j < n_in ? 1u << j : 0u;
        for (int tries = 0; left; ++tries) {
            RsPacket v[FLIGHT];  // (unconditionally: partly loaded, they would spill)
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j) v[j] = rs_peek(src + min(b0 + 32 * j, n_in - 1));
            // left, right: rows of hx; upper, lower: the plane's halo rows
            const int nL = t.n_l, nLR = t.n_lr, nLRT = t.n_lrt;
            const int oL = t.hx + 4 * par * t.nrows, oR = oL + 2 * (t.nrows - nL),
                      oT = nxt - 2 * nLR, oB = nxt + (t.nrows + 2) * t.pitch - 2 * nLRT;
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
                if (((left >> j) & 1u) && (unsigned)(v[j].a >> 32) == tag &&
                    (unsigned)(v[j].b >> 32) == tag) {
                    const int i = b0 + 32 * j;
                    const int o = 2 * i + (i < nL ? oL : (i < nLR ? oR : (i < nLRT ? oT : oB)));
                    *reinterpret_cast<float2*>(rs_smem + o) =
                        make_float2(__uint_as_float((unsigned)v[j].a),
                                    __uint_as_float((unsigned)v[j].b));
                    left &= ~(1u << j);
                }
            if (left && (tries & 1023) == 1023) {
                bool stop = *reinterpret_cast<volatile unsigned*>(err) & ERR_ABORT;
                if (!stop && tries >= RS_POLLS) {
                    atomicOr(err, ERR_DEP_TIMEOUT | ERR_ABORT);
                    stop = true;
                }
                if (stop) break;
            }
        }
        if (__any_sync(0xffffffffu, left)) return false;
    }
}

// The barrier that ends a step, from the compute warps' loop and from the halo warp's; true
// when a thread of either passes bad.
__device__ __forceinline__ bool rs_barrier(bool bad, int threads)
{
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)bad), "r"(threads)
        : "memory");
    return r != 0;
}

// many: the launch covers several shots, items[CTA] = {shot, tile}; else the one shot.
static __global__ void __launch_bounds__(RS_T, 1)
    acoustic_resident_kernel(const __grid_constant__ RsShot one, const RsShot* __restrict__ many,
                             const int2* __restrict__ items)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool halo = tid >= RS_CT;
    // the shot's record is read in every step: a copy in shared memory
    const RsShot& s = *reinterpret_cast<const RsShot*>(rs_smem + RS_TILE_FLOATS);
    const RsTile& t = rs_tile();
    if (tid < (int)sizeof(RsShot) / 4) {
        const float* from = reinterpret_cast<const float*>(many ? many + items[blockIdx.x].x : &one);
        rs_smem[RS_TILE_FLOATS + tid] = from[tid];
    }
    __syncthreads();
    RsMine m;
    {
        // ---- the tile, and this thread's units of it
        const int tile = many ? items[blockIdx.x].y : (int)blockIdx.x;
        const int gx = s.gx, gz = s.gz, w4 = (s.nx + 3) / 4, nx = s.nx, nz = s.nz;
        const int tx = tile % gx, tz = tile / gx;
        auto row0 = [&](int z) { return (int)((long long)z * nz / gz); };
        RsTile w;
        w.nx = nx;
        w.nz = nz;
        w.ldx = s.ldx;
        w.fs = s.fs;
        const int c0 = tx * w4 / gx, ncol = (tx + 1) * w4 / gx - c0;
        w.ncol = ncol;
        w.x0 = 4 * c0;
        w.z0 = row0(tz);
        const int nrows = row0(tz + 1) - w.z0, pitch = 4 * ncol;
        w.nrows = nrows;
        w.pitch = pitch;
        w.left = tx > 0;
        w.right = tx < gx - 1;
        int sp = RS_PLANE0;
        auto place = [&](int floats) {
            const int o = sp;
            sp += floats;
            return o;
        };
        w.plane[0] = place((nrows + 4) * pitch);
        w.plane[1] = place((nrows + 4) * pitch);
        w.hx = place(8 * nrows);
        w.inj = place(2 * pitch);
        w.fx = place(pitch);
        w.rk = place(pitch);
        w.fz = place((nrows + 3) / 4 * 4);
        w.ring = place(12);
        w.injs = place(2);
        w.pre = place(2);
        w.tm = place(1);
        w.next = place(2);
        w.dx2 = s.inv_dx2;
        w.dz2 = s.inv_dz2;
        w.z = s.minus_zero;
        const bool has_rec = s.n_rec > 0 && s.rec_iz >= w.z0 && s.rec_iz < w.z0 + nrows;
        w.rec_row = has_rec ? s.rec_iz - w.z0 : -1;
        const bool has_src = s.src_ix >= w.x0 && s.src_ix < w.x0 + pitch && s.src_iz >= w.z0 &&
                             s.src_iz < w.z0 + nrows;
        w.src_row = has_src ? s.src_iz - w.z0 : -1;
        w.src_x = has_src ? s.src_ix - w.x0 : -1;
        w.mirror = s.fs && !s.adjoint && w.z0 == 0 ? 2 : -1;  // (a tile has 4 rows or more)
        // packets of one slot of one tile; a tile's slot holds the packets from its left,
        // right, upper and lower neighbour, as many as it has
        const int half = 2 * s.maxr + 8 * s.maxc;
        w.half = half;
        w.in = tile * 2 * half;
        w.n_l = tx > 0 ? nrows : 0;
        w.n_lr = w.n_l + (tx < gx - 1 ? nrows : 0);
        w.n_lrt = w.n_lr + (tz > 0 ? 4 * ncol : 0);
        w.n_in = w.n_lrt + (tz < gz - 1 ? 4 * ncol : 0);
        rs_interior(nrows, ncol, &w.nci, &w.nseg, &w.R);
        if (tid == 0) *reinterpret_cast<RsTile*>(rs_smem) = w;

        if (warp == RS_CT / 32) {  // the halo warp: 512 columns, the whole tensor memory
            tm_converge();
            asm volatile(
                "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                    smem_u32(rs_smem + w.tm))
                : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::
                             : "memory");
        }
        // sponge factors by column and by row, receivers by column
        const int n = s.n_sponge;
        for (int c = tid; c < pitch; c += RS_T) {
            const int ix = w.x0 + c;
            const int d = min(n, max(0, max(n - ix, ix - (nx - 1 - n))));
            rs_smem[w.fx + c] = s.lut && d > 0 ? s.lut[d] : 1.0f;
            int r = -1;
            if (has_rec && ix < nx) {
                if (s.rec_c0 >= 0) {
                    const int q = ix - s.rec_c0;
                    r = q >= 0 && q < s.n_rec ? q : -1;
                } else {
                    const int a = s.rec_ptr[ix];
                    r = s.rec_ptr[ix + 1] > a ? s.rec_list[a] : -1;
                }
            }
            rs_smem[w.rk + c] = __int_as_float(r);
        }
        for (int r = tid; r < nrows; r += RS_T) {
            const int iz = w.z0 + r;
            const int d = min(n, max(0, max(iz - (nz - 1 - n), s.fs ? 0 : n - iz)));
            rs_smem[w.fz + r] = s.lut && d > 0 ? s.lut[d] : 1.0f;
        }

        m.ox = m.oz = -1;
        m.e = 0;
        int er = 0, ec = 0;
        const bool e_live = !halo && tid < 2 * nrows + 4 * (ncol - 2);
        if (e_live) {
            if (tid < 2 * nrows) {
                ec = tid < nrows ? 0 : ncol - 1;
                er = tid < nrows ? tid : tid - nrows;
            } else {
                const int v = tid - 2 * nrows, q = v / (ncol - 2);
                ec = 1 + v - q * (ncol - 2);
                er = q < 2 ? q : nrows - 4 + q;
            }
            // where the unit's packets go: its place in the neighbour's slot
            auto from_z = [&](int z, bool upper) {  // tile row z's upper / lower packets
                const int q = (row0(z + 1) - row0(z)) * ((tx > 0) + (tx < gx - 1));
                return upper ? q : q + (z > 0 ? 4 * ncol : 0);
            };
            if (ec == 0 && tx > 0) m.ox = (tile - 1) * 2 * half + (tx > 1 ? nrows : 0) + er;
            if (ec == ncol - 1 && tx < gx - 1) m.ox = (tile + 1) * 2 * half + er;
            if (er < 2 && tz > 0)
                m.oz = (tile - gx) * 2 * half + from_z(tz - 1, false) + er * 2 * ncol + 2 * ec;
            if (er >= nrows - 2 && tz < gz - 1)
                m.oz = (tile + gx) * 2 * half + from_z(tz + 1, true) +
                       (er - (nrows - 2)) * 2 * ncol + 2 * ec;
        }
        auto has_rule = [&](int row, int c) {
            return row == w.rec_row || (row == w.src_row && c == w.src_x >> 2) || row == w.mirror;
        };
        const bool e_write = e_live && w.z0 + er >= 2 && w.z0 + er < nz - 2;
        m.e = (unsigned)er | (unsigned)ec << 16 | (unsigned)e_live << 31 |
              (unsigned)e_write << 30 | (unsigned)(e_write && has_rule(er, ec)) << 29 |
              (unsigned)(ec == ncol - 1) << 28;
        const bool live = !halo && tid < w.nci * w.nseg;
        const int seg = live ? tid / w.nci : 0;
        const int ic = live ? 1 + tid - seg * w.nci : 1, r0 = 2 + seg * w.R;
        const int n_rows = live ? min(w.R, nrows - 2 - r0) : 0;
        m.h = (unsigned)(w.hx + 2 * er + (ec == 0 ? 0 : 2 * nrows)) | (unsigned)(4 * nrows) << 16;
        m.i = (unsigned)ic | (unsigned)r0 << 8 | (unsigned)n_rows << 24;
        m.b = 0;
        for (int i = 0; i < n_rows; ++i) m.b |= has_rule(r0 + i, ic) ? 1u << i : 0u;
        for (int j = 0; j < 4; ++j) {
            const int xe = w.x0 + 4 * ec + j, xi = w.x0 + 4 * ic + j;
            m.b |= (xe >= 2 && xe < nx - 2 ? 0x10000u << j : 0u) |
                   (xi >= 2 && xi < nx - 2 ? 0x100000u << j : 0u);
        }
        __syncthreads();
        // factors of one everywhere: the warp skips them
        auto plain = [&](int c) {
            const float4 f = *reinterpret_cast<const float4*>(rs_smem + w.fx + 4 * c);
            return f.x == 1.0f && f.y == 1.0f && f.z == 1.0f && f.w == 1.0f;
        };
        bool i_fr = n_rows && (!plain(ic) || m.i_xm() != 15u);
        for (int i = 0; i < n_rows; ++i) i_fr |= rs_smem[w.fz + r0 + i] != 1.0f;
        const bool e_fr =
            e_live && (!plain(ec) || m.e_xm() != 15u || rs_smem[w.fz + er] != 1.0f);
        m.b |= (__any_sync(0xffffffffu, i_fr) ? 1u << 24 : 0u) |
               (__any_sync(0xffffffffu, e_fr) ? 1u << 25 : 0u);
        m.tm = __float_as_uint(rs_smem[w.tm]) + ((uint32_t)(warp & 3) << 21) +
               (uint32_t)((warp >> 2) & 3) * 128u;
    }
    // (a warp without edge units, or without interior ones, skips that phase)
    const bool e_warp = !halo && (tid & ~31) < 2 * t.nrows + 4 * (t.ncol - 2);
    const bool i_warp = !halo && (tid & ~31) < t.nci * t.nseg;  // the warp has interior units
    RsConst kc;
    kc.k0 = pk(-2.5f, -2.5f);
    kc.k1 = pk(4.0f / 3.0f, 4.0f / 3.0f);
    kc.k2 = pk(-1.0f / 12.0f, -1.0f / 12.0f);
    kc.dx2 = pk(t.dx2, t.dx2);
    kc.dz2 = pk(t.dz2, t.dz2);
    kc.m2 = pk(-2.0f, -2.0f);
    kc.z = pk(t.z, t.z);
    bool bad = false;
    unsigned tag = s.tag0 + 1u;
    const int pitch = t.pitch, dpl = t.plane[1] - t.plane[0];
    const bool adj_top = s.adjoint && s.fs && t.z0 == 0;

    for (int ka = s.k0; ka < s.k1 && !bad;) {
        // the steps of one pass
        const int nt = s.nt;
        const bool fwd = ka < nt;
        const int kb = fwd ? min(s.k1, nt) : s.k1;
        const int base = fwd ? 0 : 3;
        int m3 = (fwd ? ka : ka - nt) % 3;
        int par = 0;  // plane[par] is p_curr
        // what step k adds to its p_next: the next step's source sample or receiver row
        // (-0: adding it changes nothing)
        auto src_value = [&](int k) {
            return fwd && t.src_row >= 0 && k + 1 < nt ? fmul(s.wavelet[k + 1], s.dt2_inj) : -0.0f;
        };
        auto data_row = [&](int k) -> const float* {
            const int it = 2 * nt - 1 - k;
            return !fwd && it >= 1 && t.rec_row >= 0 ? s.data + (size_t)(it - 1) * s.n_rec
                                                     : nullptr;
        };
        auto rec_row_out = [&](int k) {
            return fwd && s.rec_out ? s.rec_out + (size_t)k * s.n_rec : nullptr;
        };
        // what the receiver row's data are scaled by: dt^2, or (adjoint) c s of the cell
        auto inj_factor = [&](int c) {
            if (!s.adjoint) return s.dt2_inj;
            const float v = s.vel[1][(size_t)s.rec_iz * t.ldx + t.x0 + c];
            return fmul(v, fminf(rs_smem[t.fx + c], rs_smem[t.fz + t.rec_row]));
        };
        auto rec_of = [&](int c) { return __float_as_int(rs_smem[t.rk + c]); };
        // ---- the state into the SM
        {
            const int nrows = t.nrows, ncol = t.ncol, nz = t.nz, ldx = t.ldx;
            const float* pc = s.wave[base + (m3 + 1) % 3];
            const float* pp = s.wave[base + m3];
            const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 *d0 = reinterpret_cast<float4*>(rs_smem + t.plane[0]),
                   *d1 = reinterpret_cast<float4*>(rs_smem + t.plane[1]);
#pragma unroll 4
            for (int i = tid; i < (nrows + 4) * ncol; i += RS_T) {
                const int r = i / ncol - 2, c = i - (r + 2) * ncol, iz = t.z0 + r;
                const size_t o = (size_t)iz * ldx + t.x0 + 4 * c;
                const bool in_grid = iz >= 0 && iz < nz;
                d0[i] = in_grid ? *reinterpret_cast<const float4*>(pc + o) : z4;
                d1[i] = in_grid && r >= 0 && r < nrows ? *reinterpret_cast<const float4*>(pp + o)
                                                       : z4;
            }
            float2* hx = reinterpret_cast<float2*>(rs_smem + t.hx);
            for (int r = tid; r < nrows; r += RS_T) {
                const float* row = pc + (size_t)(t.z0 + r) * ldx + t.x0;
                float2 l = make_float2(0.f, 0.f), g = l;
                if (t.left) l = *reinterpret_cast<const float2*>(row - 2);
                if (t.right) g = *reinterpret_cast<const float2*>(row + t.pitch);
                hx[r] = l;
                hx[nrows + r] = g;
                hx[2 * nrows + r] = hx[3 * nrows + r] = make_float2(0.f, 0.f);
            }
            if (tid < 2) rs_smem[t.next + tid] = __int_as_float(0);
            if (tid < 12) {
                const int b = tid >> 2, cell = tid & 3;
                const int ix = cell < 2 ? cell : t.nx - 4 + cell;
                rs_smem[t.ring + tid] =
                    t.rec_row >= 0 ? s.wave[base + b][(size_t)s.rec_iz * ldx + ix] : 0.0f;
            }
            if (!halo) {  // tensor memory: every lane of a warp takes part
                const float* vel = s.vel[fwd ? 0 : 1];
                const float* accg = fwd ? s.illum : s.image;
                auto get = [&](const float* p, bool ok, size_t o) {
                    return p && ok ? *reinterpret_cast<const float4*>(p + o)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
                };
                auto put = [&](const float4& v, int word) {
                    uint32_t r[4];
                    bits_of(v, r);
                    tm_converge();
                    tm_st4(m.tm + word, r);
                };
                const size_t eo = (size_t)(t.z0 + m.er()) * ldx + t.x0 + 4 * m.ec();
                const float4 ev = get(vel, m.e_live(), eo), ea = get(accg, m.e_live(), eo);
                put(ev, RS_TM_CE);
                put(ea, RS_TM_AE);
                if (i_warp)
                    for (int i0 = 0; i0 < t.R; i0 += 5) {  // five rows under way at a time
                        float4 v[5], a[5];
                        const size_t o = (size_t)(t.z0 + m.r0() + i0) * ldx + t.x0 + 4 * m.c();
#pragma unroll
                        for (int j = 0; j < 5; ++j) {
                            v[j] = get(vel, i0 + j < m.n(), o + (size_t)j * ldx);
                            a[j] = get(accg, i0 + j < m.n(), o + (size_t)j * ldx);
                        }
#pragma unroll
                        for (int j = 0; j < 5; ++j)
                            if (i0 + j < RS_MAXR) {
                                put(v[j], RS_TM_C + 4 * (i0 + j));
                                put(a[j], RS_TM_A + 4 * (i0 + j));
                            }
                    }
                tm_wait_st();
            } else {
                const float* d = data_row(ka);
                for (int c = lane; c < t.pitch; c += 32) {
                    const int r = rec_of(c);
                    rs_smem[t.inj + c] = d && r >= 0 ? fmul(d[r], inj_factor(c)) : -0.0f;
                }
                if (lane == 0) rs_smem[t.injs] = src_value(ka);
            }
        }
        __syncthreads();
        // this step's snapshot: ks = it / interval, and whether it is one (rem == 0)
        int ks = (fwd ? ka : 2 * nt - 1 - ka) / s.interval,
            rem = (fwd ? ka : 2 * nt - 1 - ka) - ks * s.interval;

        // one step on: roles, packet tag, this step's place between snapshots
        auto advance = [&]() {
            m3 = m3 == 2 ? 0 : m3 + 1;
            ++tag;
            par ^= 1;
            if (fwd) {
                if (++rem == s.interval) {
                    rem = 0;
                    ++ks;
                }
            } else if (rem-- == 0) {
                rem = s.interval - 1;
                --ks;
            }
        };
        if (!halo) {
#pragma unroll 1
            for (int k = ka; k < kb; ++k) {
                // nothing derived from the records or from m is kept from step to step: it
                // would not fit the registers
                asm volatile("" : "+r"(m.e), "+r"(m.i), "+r"(m.b)::"memory");
                const int cur = RS_PLANE0 + (par ? dpl : 0), nxt = RS_PLANE0 + (par ? 0 : dpl);
                const bool on = rem == 0;  // a step with a snapshot
                // ---- phase E
                if (e_warp) {
                    const int ec = m.ec(), oc = cur + (m.er() + 2) * pitch + 4 * ec;
                    uint32_t cb[4];
                    tm_converge();
                    tm_ld4(m.tm + RS_TM_CE, cb);
                    const F4 c = ld_f4(rs_smem + oc);
                    const f32x2 l = rs_pair(ec > 0 ? oc - 2 : m.hx(par)),
                                r = rs_pair(m.last_col() ? m.hx(par) : oc + 4);
                    F4 w0 = ld_f4(rs_smem + oc - 2 * pitch), w1 = ld_f4(rs_smem + oc - pitch);
                    const F4 w3 = ld_f4(rs_smem + oc + pitch),
                             w4 = ld_f4(rs_smem + oc + 2 * pitch);
                    if (adj_top && m.er() == 2) {
                        w1 = f4_neg(c);
                        w0 = f4_neg(w3);
                    }
                    float* np = rs_smem + oc + nxt - cur;
                    const F4 pp = ld_f4(np);
                    uint4* out = s.xbuf + (tag & 1u) * t.half;
                    tm_wait_ld(cb);
                    F4 lap;
                    F4 u = rs_stencil(kc, w0, w1, c, w3, w4, l, r, pp, f4_bits(cb), lap);
                    if (m.e_frame())
                        u = rs_frame(u, *reinterpret_cast<const float4*>(rs_smem + t.fx + 4 * ec),
                                     rs_smem[t.fz + m.er()], m.e_xm(), kc.z);
                    if (m.e_spec())
                        u = rs_special(u, nxt, m.er(), ec, par, m3 == 0 ? 2 : m3 - 1, m.e_xm(),
                                       pitch, !fwd && k < 2 * nt - 1);
                    float v[4];
                    f4_get(u, v);
                    if (m.ox >= 0)
                        rs_send(out + m.ox, ec == 0 ? v[0] : v[2], ec == 0 ? v[1] : v[3], tag);
                    if (m.oz >= 0) {
                        rs_send(out + m.oz, v[0], v[1], tag);
                        rs_send(out + m.oz + 1, v[2], v[3], tag);
                    }
                    if (m.e_write()) st_f4(np, u);
                    if (on && fwd && s.lap && m.e_live())
                        rs_snap(s.snaps + (size_t)(ks - s.slot0) * s.plane +
                                    (size_t)(t.z0 + m.er()) * t.ldx + t.x0 + 4 * ec, lap);
                }
                RsFused fu{nullptr, nullptr, false, false, adj_top && m.r0() == 2};
                if (on) {
                    fu.lap = fwd && s.lap;
                    if (s.snaps) {
                        float* sn = s.snaps + (size_t)(ks - s.slot0) * s.plane;
                        if (fwd) fu.snap_out = sn;
                        else if (s.image && ks < s.n_snaps) fu.snap_in = sn;
                    }
                    fu.acc = fwd ? s.illum != nullptr : fu.snap_in != nullptr;
                }
                if (e_warp && (fu.acc || fu.snap_out)) {
                    const int ec = m.ec(), er = m.er();
                    const F4 c = ld_f4(rs_smem + cur + (er + 2) * pitch + 4 * ec);
                    if (fu.snap_out && !fu.lap && m.e_live())
                        rs_snap(fu.snap_out + (size_t)(t.z0 + er) * t.ldx + t.x0 + 4 * ec, c);
                    if (fu.acc) {
                        uint32_t ab[4];
                        tm_converge();
                        tm_ld4(m.tm + RS_TM_AE, ab);
                        float4 fe = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (fu.snap_in && m.e_live())
                            fe = *reinterpret_cast<const float4*>(
                                fu.snap_in + (size_t)(t.z0 + er) * t.ldx + t.x0 + 4 * ec);
                        tm_wait_ld(ab);
                        const f32x2 dt = pk(s.img_dt, s.img_dt);
                        const F4 acc = fu.snap_in ? rs_image(f4_bits(ab), c, fe, dt, kc.z)
                                                  : rs_illum(f4_bits(ab), c, kc.z);
                        uint32_t o[4];
                        bits_f4(acc, o);
                        tm_converge();
                        tm_st4(m.tm + RS_TM_AE, o);
                        tm_wait_st();
                    }
                }
                // ---- phase I
                tm_converge();
                if (i_warp) {
                    if (fu.acc || fu.snap_out)
                        rs_inner<true>(m, kc, pitch, cur, nxt, t.R, fu, pk(s.img_dt, s.img_dt));
                    else
                        rs_inner<false>(m, kc, pitch, cur, nxt, t.R, fu, 0);
                    for (unsigned b = m.spec(); b; b &= b - 1) {
                        const int r = m.r0() + __ffs(b) - 1, c = m.c();
                        float* o = rs_smem + nxt + (r + 2) * pitch + 4 * c;
                        st_f4(o, rs_special(ld_f4(o), nxt, r, c, par, m3 == 0 ? 2 : m3 - 1,
                                            m.i_xm(), pitch, !fwd && k < 2 * nt - 1));
                    }
                    __syncwarp();
                }
                bad = !rs_collect<RS_FLIGHT_C>(s.xbuf + t.in + (tag & 1u) * t.half, tag, nxt, par ^ 1,
                                     t.next + par, s.err);
                advance();
                if (rs_barrier(bad, RS_T)) {
                    bad = true;
                    break;
                }
            }
        } else {
            // Injection values, a step ahead in registers: what a step adds is loaded during the
            // step before the last one and staged in the last one (columns lane + 32 j; those
            // of tiles wider than 256 points past them as they are staged).
            float nd[8], nf[8], ns = -0.0f;
            const bool rec = !fwd && t.rec_row >= 0;
            auto load_injection = [&](int k) {
                const float* d = k < kb ? data_row(k) : nullptr;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = lane + 32 * j, r = c < pitch ? rec_of(c) : -1;
                    nd[j] = d && r >= 0 ? d[r] : -0.0f;
                }
            };
            auto load_source = [&](int k) {
                ns = fwd && t.src_row >= 0 && k < kb && k + 1 < nt ? s.wavelet[k + 1] : -0.0f;
            };
            if (rec) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = lane + 32 * j;
                    nf[j] = c < pitch && rec_of(c) >= 0 ? inj_factor(c) : 1.0f;
                }
                load_injection(ka + 1);
            }
            load_source(ka + 1);
#pragma unroll 1
            for (int k = ka; k < kb; ++k) {
                const int cur = RS_PLANE0 + (par ? dpl : 0), nxt = RS_PLANE0 + (par ? 0 : dpl);
                const bool more = k + 1 < kb;
                if (rec) {
                    float* inj = rs_smem + t.inj + (par ^ 1) * pitch;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (lane + 32 * j < pitch) inj[lane + 32 * j] = fmul(nd[j], nf[j]);
                    load_injection(k + 2);
                    for (int c = 256 + lane; c < pitch; c += 32) {
                        const float* d = more ? data_row(k + 1) : nullptr;
                        const int r = rec_of(c);
                        inj[c] = d && r >= 0 ? fmul(d[r], inj_factor(c)) : -0.0f;
                    }
                }
                if (lane == 0) {
                    rs_smem[t.injs + (par ^ 1)] = fmul(ns, s.dt2_inj);
                    reinterpret_cast<int*>(rs_smem)[t.next + (par ^ 1)] = 0;
                }
                load_source(k + 2);
                if (k > ka && t.rec_row >= 0 && rec_row_out(k - 1))
                    rs_sample(rec_row_out(k - 1), cur, par ^ 1);
                if (!fwd && more && s.image && s.snaps && (rem == 1 || s.interval == 1)) {
                    const int k1 = rem == 0 ? ks - 1 : ks;
                    if (k1 < s.n_snaps)
                        for (int r = lane; r < t.nrows; r += 32)
                            prefetch_l2_bulk(s.snaps + (size_t)(k1 - s.slot0) * s.plane +
                                                 (size_t)(t.z0 + r) * t.ldx + t.x0,
                                             (uint32_t)t.pitch * 4u);
                }
                __syncwarp();
                bad = !rs_collect<RS_FLIGHT_H>(s.xbuf + t.in + (tag & 1u) * t.half, tag, nxt,
                                             par ^ 1, t.next + par, s.err);
                advance();
                if (rs_barrier(bad, RS_T)) {
                    bad = true;
                    break;
                }
            }
        }

        // ---- the state back to memory: p_prev and p_curr of step kb (and, on the
        // receiver row, what the third buffer holds in the never-written cells)
        if (!bad) {
            const int nrows = t.nrows, ncol = t.ncol, ldx = t.ldx;
            float* pp = s.wave[base + m3];
            float* pc = s.wave[base + (m3 + 1) % 3];
            float* p3 = s.wave[base + (m3 + 2) % 3];
            const float4* sc =
                reinterpret_cast<const float4*>(rs_smem + t.plane[par] + 2 * t.pitch);
            const float4* sv =
                reinterpret_cast<const float4*>(rs_smem + t.plane[par ^ 1] + 2 * t.pitch);
#pragma unroll 4
            for (int i = tid; i < nrows * ncol; i += RS_T) {
                const int r = i / ncol, c = i - r * ncol;
                const size_t o = (size_t)(t.z0 + r) * ldx + t.x0 + 4 * c;
                *reinterpret_cast<float4*>(pc + o) = sc[i];
                *reinterpret_cast<float4*>(pp + o) = sv[i];
            }
            if (halo && t.rec_row >= 0 && rec_row_out(kb - 1))
                rs_sample(rec_row_out(kb - 1), RS_PLANE0 + (par ? dpl : 0), par ^ 1);
            if (t.rec_row >= 0 && tid < 4) {
                const int ix = tid < 2 ? tid : t.nx - 4 + tid;
                if (ix >= t.x0 && ix < t.x0 + t.pitch)
                    p3[(size_t)s.rec_iz * ldx + ix] = rs_smem[t.ring + 4 * ((m3 + 2) % 3) + tid];
            }
            float* accg = fwd ? s.illum : s.image;
            if (!halo && accg) {
                auto get = [&](bool ok, size_t o, int word) {
                    uint32_t r[4];
                    tm_converge();
                    tm_ld4(m.tm + word, r);
                    tm_wait_ld(r);
                    if (ok)
                        *reinterpret_cast<float4*>(accg + o) =
                            make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]),
                                        __uint_as_float(r[2]), __uint_as_float(r[3]));
                };
                get(m.e_live(), (size_t)(t.z0 + m.er()) * ldx + t.x0 + 4 * m.ec(), RS_TM_AE);
                if (i_warp)
                    for (int i = 0; i < t.R; ++i)
                        get(i < m.n(), (size_t)(t.z0 + m.r0() + i) * ldx + t.x0 + 4 * m.c(),
                            RS_TM_A + 4 * i);
            }
            __syncthreads();
        }
        ka = kb;
    }
    __syncthreads();
    if (warp == RS_CT / 32) {
        tm_converge();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(
                         __float_as_uint(rs_smem[t.tm]))
                     : "memory");
    }
}

cudaError_t launch_acoustic_resident(const RsShot& one, const RsShot* many, const int2* items,
                                     int ctas, cudaStream_t st)
{
    const cudaError_t e = set_smem_once<acoustic_resident_kernel>(RS_SMEM);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(RS_T);
    cfg.dynamicSmemBytes = RS_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, acoustic_resident_kernel, one, many, items);
}

int rs_capacity()
{
    // one query per device, safe when several host threads ask
    auto query = [](int dev) {
        int coop = 0, sms = 0, per = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
            !coop ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            set_smem_once<acoustic_resident_kernel>(RS_SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, acoustic_resident_kernel, RS_T,
                                                          RS_SMEM) != cudaSuccess)
            return 0;
        return per > 0 ? sms : 0;
    };
    static std::once_flag once[W2D_MAX_DEVICES];
    static int cap[W2D_MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < 0 || dev >= W2D_MAX_DEVICES) return query(dev);
    std::call_once(once[dev], [&query, dev] { cap[dev] = query(dev); });
    return cap[dev];
}

}  // namespace w2d

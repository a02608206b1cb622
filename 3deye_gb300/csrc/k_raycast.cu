// k_raycast.cu -- model prediction: TSDF ray march (raycast), model-map
// pyramid (resize) and rigid map transform.
//
// Built with -fmad=false: every float expression below is evaluated as the
// same sequence of IEEE-rounded multiplies and adds the reference kernel
// (GPU/opencl/raycast.cl) performs, so vertex/normal maps match the
// reference bit for bit on the same volume.
#include "tde_common.cuh"
#include "tde_launch.cuh"
#include "tde_integrate.cuh"

namespace tde {
namespace {

struct RayParams {
    tde_point3f t;          // ray origin (camera centre, volume frame)
    tde_matrix3f R;         // camera -> volume rotation
    float time_step;        // (float)((double)trunc * 0.8), raycast.cl:209
    float max_time;         // 3 * (Vx + Vy + Vz), raycast.cl:251
    tde_intrinsics intr;
    tde_round_buffer rb;
    tde_point3f cell;
    size_t n;               // voxel count (F32 plane offset)
    const CamPose *dpose;   // when set, t and R are read from here
    const uint8_t *neg_flags;  // per physical 8^3 brick: 0 = holds no negative value
    const uint8_t *super_flags;  // per physical 32^3 super-brick (whole ones only)
    const unsigned long long *neg_masks;  // the brick flags as one word per super-brick (FLAG_MASKS)
    float inv_cell[3];
    unsigned *touched;      // measurement runs: one bit per voxel record read
};

struct f3 { float x, y, z; };

__device__ __forceinline__ f3 mat_vec(const tde_matrix3f &M, f3 v) {
    // multiply() in elementary_matrix_template.h:30-39: dot starting from 0.
    f3 r;
    float a = 0.f; a += M.row[0].x * v.x; a += M.row[0].y * v.y; a += M.row[0].z * v.z; r.x = a;
    float b = 0.f; b += M.row[1].x * v.x; b += M.row[1].y * v.y; b += M.row[1].z * v.z; r.y = b;
    float c = 0.f; c += M.row[2].x * v.x; c += M.row[2].y * v.y; c += M.row[2].z * v.z; r.z = c;
    return r;
}

__device__ __forceinline__ f3 normalized(f3 v) {
    float d = 0.f; d += v.x * v.x; d += v.y * v.y; d += v.z * v.z;
    float rs = 1.f / sqrtf(d);
    return f3{v.x * rs, v.y * rs, v.z * rs};
}

// ray_start + ray_dir * t, component-wise (add_3f after the scale).
__device__ __forceinline__ f3 along(f3 o, f3 d, float t) {
    return f3{o.x + d.x * t, o.y + d.y * t, o.z + d.z * t};
}

__device__ __forceinline__ int floor_sat(float v) { return __float2int_rd(v); }  // convert_int_sat_rtn

// A voxel record's value; measurement instantiations also mark the record.
template <int FMT, bool STATS>
__device__ __forceinline__ float load_rec(const void *vol, const RayParams &p, size_t addr) {
    if (STATS) atomicOr(p.touched + (addr >> 5), 1u << (addr & 31));
    return TsdfStore<FMT>::value(vol, addr, p.n);
}

template <int FMT, bool STATS>
__device__ __forceinline__ float read_tsdf(const void *vol, const RayParams &p, int x, int y, int z) {
    return load_rec<FMT, STATS>(vol, p, voxel_address(x, y, z, p.rb));
}

// interpolateTrilineary (raycast.cl:95-145), split by axis: the lower corner
// along one axis, the upper corner's weight, and both corners' physical
// indices times the axis stride.  False when the base voxel lies on the
// volume border (the interpolation is then NaN).  The six normal samples of a
// hit share two of their three axes with the refined point, so those are
// formed once.
struct Axis {
    unsigned i0, i1;  // a volume has fewer than 2^31 voxels
    float w;
};

__device__ __forceinline__ bool tri_axis(float pt, float q, float cell, int N, int origin, unsigned stride, Axis &ax) {
    int g = floor_sat(q);
    if (g <= 0 || g >= N - 1) return false;
    const float v = ((float)g + 0.5f) * cell;
    g = (pt < v) ? g - 1 : g;
    float a = q - ((float)g + 0.5f);
    if (a < 0) { g--; a += 1.0f; }
    // the two corners g, g + 1 are inside [0, N) here, and so is the origin
    const int w0 = g + origin, w1 = w0 + 1;
    ax.i0 = (unsigned)(w0 - (w0 >= N ? N : 0)) * stride;
    ax.i1 = (unsigned)(w1 - (w1 >= N ? N : 0)) * stride;
    ax.w = a;
    return true;
}

template <int FMT, bool STATS>
__device__ __forceinline__ float tri_corners(const void *vol, const RayParams &p, const Axis &X, const Axis &Y,
                                             const Axis &Z) {
    const unsigned r00 = Y.i0 + Z.i0, r01 = Y.i0 + Z.i1, r10 = Y.i1 + Z.i0, r11 = Y.i1 + Z.i1;
    float v000 = load_rec<FMT, STATS>(vol, p, X.i0 + r00), v001 = load_rec<FMT, STATS>(vol, p, X.i0 + r01);
    float v010 = load_rec<FMT, STATS>(vol, p, X.i0 + r10), v011 = load_rec<FMT, STATS>(vol, p, X.i0 + r11);
    float v100 = load_rec<FMT, STATS>(vol, p, X.i1 + r00), v101 = load_rec<FMT, STATS>(vol, p, X.i1 + r01);
    float v110 = load_rec<FMT, STATS>(vol, p, X.i1 + r10), v111 = load_rec<FMT, STATS>(vol, p, X.i1 + r11);
    const float a = X.w, b = Y.w, c = Z.w;
    float one_a = 1.f - a, one_b = 1.f - b, one_c = 1.f - c;
    float xa = one_b * (v000 * one_c + v001 * c) + b * (v010 * one_c + v011 * c);
    float xb = one_b * (v100 * one_c + v101 * c) + b * (v110 * one_c + v111 * c);
    return one_a * xa + a * xb;
}

__device__ __forceinline__ bool axis_x(const RayParams &p, float pt, float q, Axis &ax) {
    return tri_axis(pt, q, p.cell.x, p.rb.voxels_size.x, p.rb.origin_GRID.x, 1, ax);
}
__device__ __forceinline__ bool axis_y(const RayParams &p, float pt, float q, Axis &ax) {
    return tri_axis(pt, q, p.cell.y, p.rb.voxels_size.y, p.rb.origin_GRID.y, (unsigned)p.rb.voxels_size.x, ax);
}
__device__ __forceinline__ bool axis_z(const RayParams &p, float pt, float q, Axis &ax) {
    return tri_axis(pt, q, p.cell.z, p.rb.voxels_size.z, p.rb.origin_GRID.z,
                    (unsigned)p.rb.voxels_size.x * (unsigned)p.rb.voxels_size.y, ax);
}

// Zero crossing between time_curr and time_curr + step: secant refinement of
// the hit and central-difference normal (raycast.cl:280-401).  Kept out of
// line: it runs once per ray, and inlining it would bloat the march loop past
// the instruction cache.  The samples' places are settled before their values
// are read, so the reads of the two march samples, and then of the six normal
// samples, are in flight together; a sample on the volume's border makes the
// point, or the normal, NaN as a whole.
template <int FMT, bool STATS>
__device__ __noinline__ void refine_surface(const void *vol, const RayParams &p, f3 org, f3 dir, float time_curr,
                                            float &vx_out, float &vy_out, float &vz_out, float &nx_out,
                                            float &ny_out, float &nz_out) {
    const tde_point3i N = p.rb.voxels_size;
    const float step = p.time_step;
    const f3 pa = along(org, dir, time_curr + step), pb = along(org, dir, time_curr);
    const f3 qb{pb.x / p.cell.x, pb.y / p.cell.y, pb.z / p.cell.z};
    Axis X, Y, Z, X2, Y2, Z2;
    if (!axis_x(p, pa.x, pa.x / p.cell.x, X) || !axis_y(p, pa.y, pa.y / p.cell.y, Y) ||
        !axis_z(p, pa.z, pa.z / p.cell.z, Z))
        return;
    // (a measurement reads as the reference does: one after the other)
    if (STATS && isnan(tri_corners<FMT, STATS>(vol, p, X, Y, Z))) return;
    if (!axis_x(p, pb.x, qb.x, X2) || !axis_y(p, pb.y, qb.y, Y2) || !axis_z(p, pb.z, qb.z, Z2)) return;
    const float Ftdt = tri_corners<FMT, STATS>(vol, p, X, Y, Z);
    const float Ft = tri_corners<FMT, STATS>(vol, p, X2, Y2, Z2);
    if (isnan(Ftdt) || isnan(Ft)) return;
    float Ts = time_curr - step * Ft / (Ftdt - Ft);
    f3 vf = along(org, dir, Ts);
    vx_out = vf.x; vy_out = vf.y; vz_out = vf.z;
    int hx = floor_sat(qb.x), hy = floor_sat(qb.y), hz = floor_sat(qb.z);
    if (hx > 1 && hy > 1 && hz > 1 && hx < N.x - 2 && hy < N.y - 2 && hz < N.z - 2) {
        // vf +- cell on one axis: the other two axes are vf's
        Axis P1, P2, Q1, Q2, R1, R2;
        const bool okx = axis_x(p, vf.x, vf.x / p.cell.x, X);
        const bool oky = axis_y(p, vf.y, vf.y / p.cell.y, Y);
        const bool okz = axis_z(p, vf.z, vf.z / p.cell.z, Z);
        float t1 = vf.x + p.cell.x, t2 = vf.x - p.cell.x;
        const bool x1 = axis_x(p, t1, t1 / p.cell.x, P1), x2 = axis_x(p, t2, t2 / p.cell.x, P2);
        t1 = vf.y + p.cell.y; t2 = vf.y - p.cell.y;
        const bool y1 = axis_y(p, t1, t1 / p.cell.y, Q1), y2 = axis_y(p, t2, t2 / p.cell.y, Q2);
        t1 = vf.z + p.cell.z; t2 = vf.z - p.cell.z;
        const bool z1 = axis_z(p, t1, t1 / p.cell.z, R1), z2 = axis_z(p, t2, t2 / p.cell.z, R2);
        if (!(okx && oky && okz && x1 && x2 && y1 && y2 && z1 && z2)) {
            if (STATS) {
                if (x1 && oky && okz) tri_corners<FMT, STATS>(vol, p, P1, Y, Z);
                if (x2 && oky && okz) tri_corners<FMT, STATS>(vol, p, P2, Y, Z);
                if (okx && y1 && okz) tri_corners<FMT, STATS>(vol, p, X, Q1, Z);
                if (okx && y2 && okz) tri_corners<FMT, STATS>(vol, p, X, Q2, Z);
                if (okx && oky && z1) tri_corners<FMT, STATS>(vol, p, X, Y, R1);
                if (okx && oky && z2) tri_corners<FMT, STATS>(vol, p, X, Y, R2);
            }
            return;
        }
        const float Fx1 = tri_corners<FMT, STATS>(vol, p, P1, Y, Z), Fx2 = tri_corners<FMT, STATS>(vol, p, P2, Y, Z);
        const float Fy1 = tri_corners<FMT, STATS>(vol, p, X, Q1, Z), Fy2 = tri_corners<FMT, STATS>(vol, p, X, Q2, Z);
        const float Fz1 = tri_corners<FMT, STATS>(vol, p, X, Y, R1), Fz2 = tri_corners<FMT, STATS>(vol, p, X, Y, R2);
        f3 n = normalized(f3{Fx1 - Fx2, Fy1 - Fy2, Fz1 - Fz2});
        nx_out = n.x; ny_out = n.y; nz_out = n.z;
    }
}

// Voxel of the sample at time ct: floor(pos / cell) with pos = t + dir * ct
// evaluated exactly as the reference does whenever it matters.  With u = 2^-24
// and M = |o/c| + |d/c| ct, the estimate o/c + (d/c) ct is within 6 u M of the
// reference's quotient (two roundings each of o/c and d/c and one of the sum; the
// reference's product, sum and quotient), so an estimate further than 8 u M from
// the nearest integer settles the floor; otherwise the position and the IEEE
// quotient are computed.  The margin is formed once a ray, for the time at which
// it leaves the volume: near 5e-4 voxel in 512^3, where one warp in ten needs the
// exact form for some lane (a fixed 4e-3: every second one).
constexpr float kSkipMargin = 1e-2f;  // voxels

struct RayFast {
    float o[3], d[3];  // t / cell, dir / cell
    float inv_d[3];    // 1 / d
    float margin;      // voxels
};

// Time at which the ray (fast coordinates) leaves the box [lo, lo + size)
// shrunk by kSkipMargin voxels on every side: the last time a sample may take
// and still lie inside the box (the fast coordinates' error is far below the
// margin).
__device__ __forceinline__ float box_exit(const RayFast &rf, float lox, float loy, float loz, float sx, float sy,
                                         float sz) {
    const float ex = ((rf.d[0] > 0.f ? lox + (sx - kSkipMargin) : lox + kSkipMargin) - rf.o[0]) * rf.inv_d[0];
    const float ey = ((rf.d[1] > 0.f ? loy + (sy - kSkipMargin) : loy + kSkipMargin) - rf.o[1]) * rf.inv_d[1];
    const float ez = ((rf.d[2] > 0.f ? loz + (sz - kSkipMargin) : loz + kSkipMargin) - rf.o[2]) * rf.inv_d[2];
    return fminf(fminf(ex, ey), ez);
}

// Out of line: the march loop has to stay within the instruction cache.
__device__ __noinline__ int axis_exact(float o, float d, float cell, float ct) {
    return floor_sat((o + d * ct) / cell);
}

// Nearest integer of q (|q| < 2^22) and q's distance from it; the floor follows.
__device__ __forceinline__ int axis_floor(float q, float &dist) {
    const float magic = 12582912.f;  // 1.5 * 2^23
    const float t = q + magic;
    dist = q - (t - magic);
    return __float_as_int(t) - __float_as_int(magic) - (dist < 0.f ? 1 : 0);
}

__device__ __forceinline__ void sample_voxel(const RayParams &p, const f3 &org, const f3 &dir, const RayFast &rf,
                                             float ct, int &sx, int &sy, int &sz) {
    float dx, dy, dz;
    sx = axis_floor(fmaf(rf.d[0], ct, rf.o[0]), dx);
    sy = axis_floor(fmaf(rf.d[1], ct, rf.o[1]), dy);
    sz = axis_floor(fmaf(rf.d[2], ct, rf.o[2]), dz);
    if (!(fabsf(dx) > rf.margin && fabsf(dy) > rf.margin && fabsf(dz) > rf.margin)) {
        if (!(fabsf(dx) > rf.margin)) sx = axis_exact(org.x, dir.x, p.cell.x, ct);
        if (!(fabsf(dy) > rf.margin)) sy = axis_exact(org.y, dir.y, p.cell.y, ct);
        if (!(fabsf(dz) > rf.margin)) sz = axis_exact(org.z, dir.z, p.cell.z, ct);
    }
}

// The last of the sample times tn, tn + step, ... (each a rounded addition) before
// `lim` that a march from tn reaches before max_time; four additions a round.
__device__ __forceinline__ float advance(float tn, float step, float lim, float max_time) {
    for (;;) {
        const float a = tn + step, b = a + step, c = b + step, d = c + step;
        if (d < lim && c < max_time) { tn = d; continue; }
        // the times grow: each condition holds only where the one before does
        return (c < lim && b < max_time) ? c : (b < lim && a < max_time) ? b : (a < lim && tn < max_time) ? a : tn;
    }
}

// A block is a row of kRayWarps warps, a warp an 8 x 4 tile of pixels, so its rays
// start close together and sample neighbouring voxels.  What bounds the kernel
// at 640x480 / 512^3: its instructions (4000 a warp, 1600 of them the refinement's;
// two thirds of the issue slots while an SM is busy) and the longest rays' chain of
// loads (an SM is busy for 100 to 140 thousand cycles; blocks of 1 to 8 warps end
// within 5 % of each other).  The pipeline's cast: 97 us with byte flags read
// sample by sample; 67 us with a word of flags a super-brick, rarer exact places
// and four additions a round of `advance`; 63 us with strides across eight empty
// bricks; 61 us with the refinement's reads together.
constexpr int kRayWarps = 4;
constexpr int kRayThreads = 32 * kRayWarps;
constexpr int kRayBlockCols = 8 * kRayWarps, kRayBlockRows = 4;

// What the march knows of empty bricks: nothing, a byte each (the flags a caller
// keeps), or a word of 64 bits per 32^3 super-brick (the pipeline's): one load where
// a ray enters the super-brick in place of two dependent ones and one for each of
// its bricks.
enum FlagKind { FLAG_NONE, FLAG_BYTES, FLAG_MASKS };
// Blocks an SM holds: without flags the march waits for records and wants warps
// (86 us with 9, 93 with 7), with them the refinement's reads want registers (61 us
// with 7, 64 with 9).
constexpr int ray_blocks(FlagKind flags) { return flags == FLAG_NONE ? 9 : 7; }

// WHOLE: every axis is whole super-bricks, which strides across more than a brick
// need.  (Asked of the parameters at each stride it cost a 640x480 frame of a 512^3
// pipeline 1 us.)
template <int FMT, FlagKind FLAGS, bool WHOLE, bool STATS>
__global__ void __launch_bounds__(kRayThreads, ray_blocks(FLAGS))
    raycast_kernel(const void *vol, float *vmap, float *nmap, const __grid_constant__ RayParams p) {
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    allow_next_kernel();
    wait_previous_kernel();
    const int x = blockIdx.x * kRayBlockCols + warp * 8 + (lane & 7);
    const int y = (int)(blockIdx.z * gridDim.y + blockIdx.y) * kRayBlockRows + (lane >> 3);
    const int W = p.intr.cols, H = p.intr.rows;
    // the pose: from the parameters, or read on the device
    tde_matrix3f R = p.R;
    f3 org{p.t.x, p.t.y, p.t.z};
    if (p.dpose) {
        __shared__ float s_pose[12];
        if (tid < 12) s_pose[tid] = tid < 9 ? p.dpose->R[tid] : p.dpose->t[tid - 9];
        __syncthreads();
        R = tde_matrix3f{{{s_pose[0], s_pose[1], s_pose[2]}, {s_pose[3], s_pose[4], s_pose[5]},
                          {s_pose[6], s_pose[7], s_pose[8]}}};
        org = f3{s_pose[9], s_pose[10], s_pose[11]};
    }
    const float qnan = __int_as_float(0x7fffffff);
    const tde_point3i N = p.rb.voxels_size;
    const tde_point3f V = p.rb.volume_size;
    const float step = p.time_step;
    // lanes outside the image stay (no early return): the warp reconverges
    // before the refinement
    const bool inside = x < W && y < H;
    float vx_out = qnan, vy_out = qnan, vz_out = qnan;
    float nx_out = qnan, ny_out = qnan, nz_out = qnan;

    f3 rnu{((float)x - p.intr.cx) / p.intr.fx, ((float)y - p.intr.cy) / p.intr.fy, 1.f};
    f3 rn2 = mat_vec(R, rnu);
    f3 ray_next{rn2.x + org.x, rn2.y + org.y, rn2.z + org.z};
    f3 dir = normalized(f3{ray_next.x - org.x, ray_next.y - org.y, ray_next.z - org.z});
    dir.x = (dir.x == 0.f) ? 1e-15f : dir.x;
    dir.y = (dir.y == 0.f) ? 1e-15f : dir.y;
    dir.z = (dir.z == 0.f) ? 1e-15f : dir.z;

    // getMinTime / getMaxTime: raycast.cl:153-171
    float txmin = ((dir.x > 0 ? 0.f : V.x) - org.x) / dir.x;
    float tymin = ((dir.y > 0 ? 0.f : V.y) - org.y) / dir.y;
    float tzmin = ((dir.z > 0 ? 0.f : V.z) - org.z) / dir.z;
    float t_start = cl_fmax(cl_fmax(txmin, tymin), tzmin);
    float txmax = ((dir.x > 0 ? V.x : 0.f) - org.x) / dir.x;
    float tymax = ((dir.y > 0 ? V.y : 0.f) - org.y) / dir.y;
    float tzmax = ((dir.z > 0 ? V.z : 0.f) - org.z) / dir.z;
    float t_exit = cl_fmin(cl_fmin(txmax, tymax), tzmax);
    t_start = cl_fmax(t_start, 0.f);

    // the march finds the zero crossing; the secant refinement and the normal
    // run after it, once per warp for all lanes that hit (lanes reaching the
    // crossing at different samples would otherwise refine one by one)
    bool hit = false;
    float hit_time = 0.f;
    if (inside && !(t_start >= t_exit)) {
        float time_curr = t_start;
        f3 pu = along(org, dir, time_curr);
        int gx = floor_sat(pu.x / p.cell.x), gy = floor_sat(pu.y / p.cell.y), gz = floor_sat(pu.z / p.cell.z);
        gx = max(0, min(gx, N.x - 1));
        gy = max(0, min(gy, N.y - 1));
        gz = max(0, min(gz, N.z - 1));
        RayFast rf;
        rf.o[0] = org.x * p.inv_cell[0]; rf.o[1] = org.y * p.inv_cell[1]; rf.o[2] = org.z * p.inv_cell[2];
        rf.d[0] = dir.x * p.inv_cell[0]; rf.d[1] = dir.y * p.inv_cell[1]; rf.d[2] = dir.z * p.inv_cell[2];
        rf.inv_d[0] = 1.f / rf.d[0]; rf.inv_d[1] = 1.f / rf.d[1]; rf.inv_d[2] = 1.f / rf.d[2];
        // samples up to one step past the exit are placed; none of an estimate too large for axis_floor
        const float t_far = t_exit + 2.f * step;
        const float far = fmaxf(fmaxf(fmaf(fabsf(rf.d[0]), t_far, fabsf(rf.o[0])),
                                      fmaf(fabsf(rf.d[1]), t_far, fabsf(rf.o[1]))),
                                fmaf(fabsf(rf.d[2]), t_far, fabsf(rf.o[2])));
        rf.margin = far < 4194304.f ? far * 4.76837158e-7f : 1.f;  // 8 * 2^-24
        // previous sample: its value when `known`, else only "non-negative";
        // its time lets the value be fetched when it turns out to matter
        float tsdf = read_tsdf<FMT, STATS>(vol, p, gx, gy, gz);
        bool known = true;
        float prev_ct = time_curr;
        const int nbx = (N.x + 7) >> 3, nby = (N.y + 7) >> 3;
        const int nsx = (N.x + 31) >> 5, nsy = (N.y + 31) >> 5;
        int last_super = -1;

        // raycast.cl:254-404
        if (FLAGS == FLAG_NONE) {
            // kAhead samples a round: their records are read together (the next
            // sample's place does not depend on them), then tested in order: 88 us
            // at 640x480 / 512^3 for 107 one by one (3: 89, 6: 90, 8: 91)
            constexpr int kAhead = STATS ? 1 : 4;
            bool more = true;
            while (more) {
                float at[kAhead + 1], v[kAhead];
                bool alive[kAhead];
                at[0] = time_curr;
                #pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    at[k + 1] = at[k] + step;
                    int sx, sy, sz;
                    sample_voxel(p, org, dir, rf, at[k + 1], sx, sy, sz);
                    alive[k] = (k == 0 || alive[k > 0 ? k - 1 : 0]) && at[k] < p.max_time &&
                               (unsigned)sx < (unsigned)N.x && (unsigned)sy < (unsigned)N.y &&
                               (unsigned)sz < (unsigned)N.z;
                    v[k] = 0.f;
                    if (alive[k]) {
                        int px = sx + p.rb.origin_GRID.x; px -= px >= N.x ? N.x : 0;
                        int py = sy + p.rb.origin_GRID.y; py -= py >= N.y ? N.y : 0;
                        int pz = sz + p.rb.origin_GRID.z; pz -= pz >= N.z ? N.z : 0;
                        v[k] = load_rec<FMT, STATS>(
                            vol, p, (unsigned)px + (unsigned)N.x * ((unsigned)py + (unsigned)N.y * (unsigned)pz));
                    }
                }
                #pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    more = more && alive[k];
                    if (more && tsdf > 0.f && v[k] < 0.f) { hit = true; hit_time = at[k]; more = false; }
                    if (tsdf < 0.f && v[k] > 0.f) more = false;
                    tsdf = v[k];
                }
                time_curr = at[kAhead];
            }
        }
        // with flags, one sample per iteration; a sample in a super-brick (or else
        // in a brick) without negative values, after a non-negative one, lets
        // time advance by the same additions, without evaluating samples, until
        // the next one nears the exit: no test can fire in between
        unsigned long long mask = 0;
        bool empty_super = false;
        while (FLAGS != FLAG_NONE && time_curr < p.max_time) {
            const float ct = time_curr + step;
            int sx, sy, sz;
            sample_voxel(p, org, dir, rf, ct, sx, sy, sz);
            if (!((unsigned)sx < (unsigned)N.x && (unsigned)sy < (unsigned)N.y && (unsigned)sz < (unsigned)N.z)) break;
            int px = sx + p.rb.origin_GRID.x; px -= px >= N.x ? N.x : 0;
            int py = sy + p.rb.origin_GRID.y; py -= py >= N.y ? N.y : 0;
            int pz = sz + p.rb.origin_GRID.z; pz -= pz >= N.z ? N.z : 0;
            const int sid = (px >> 5) + nsx * ((py >> 5) + nsy * (pz >> 5));
            bool have, empty_eight = false;
            if (FLAGS == FLAG_MASKS) {
                if (sid != last_super) {
                    mask = p.neg_masks[sid];
                    empty_super = WHOLE && mask == 0;
                }
                have = (mask >> (((px >> 3) & 3) | ((py >> 1) & 12) | ((pz << 1) & 48))) & 1;
                // the eight bricks of the 16^3 corner of the super-brick that the sample is in
                const int corner = ((px >> 3) & 2) | ((py >> 1) & 8) | ((pz << 1) & 32);
                empty_eight = WHOLE && ((mask >> corner) & 0x330033ull) == 0;
            } else {
                if (WHOLE && sid != last_super) empty_super = !p.super_flags[sid];
                have = !empty_super && p.neg_flags[(px >> 3) + nbx * ((py >> 3) + nby * (pz >> 3))] != 0;
            }
            last_super = sid;
            if (!have && !(known && tsdf < 0.f)) {
                const int edge = empty_super ? 31 : empty_eight ? 15 : 7;
                float bx = (float)(edge + 1), by = bx, bz = bx;
                if (!WHOLE) {
                    // the last brick of an axis that is not whole bricks is shorter, and
                    // across the origin another one's voxels follow it inside the volume
                    bx = fminf(bx, (float)(N.x - (px & ~7)));
                    by = fminf(by, (float)(N.y - (py & ~7)));
                    bz = fminf(bz, (float)(N.z - (pz & ~7)));
                }
                const float lim = box_exit(rf, (float)(sx - (px & edge)), (float)(sy - (py & edge)),
                                           (float)(sz - (pz & edge)), bx, by, bz);
                time_curr = advance(ct, step, lim, p.max_time);
                known = false;
                prev_ct = time_curr;
                continue;
            }
            const unsigned addr = (unsigned)px + (unsigned)N.x * ((unsigned)py + (unsigned)N.y * (unsigned)pz);
            const float cur = load_rec<FMT, STATS>(vol, p, addr);
            if (!known) {
                if (!(cur < 0.f)) {  // prev >= 0 and cur >= 0
                    tsdf = cur;
                    known = true;
                    prev_ct = ct;
                    time_curr = ct;
                    continue;
                }
                // the previous sample's sign decides a crossing: fetch it
                int qx, qy, qz;
                sample_voxel(p, org, dir, rf, prev_ct, qx, qy, qz);
                tsdf = read_tsdf<FMT, STATS>(vol, p, qx, qy, qz);
            }
            const float tsdf_prev = tsdf;
            tsdf = cur;
            known = true;
            prev_ct = ct;
            if (tsdf_prev < 0.f && tsdf > 0.f) break;
            if (tsdf_prev > 0.f && tsdf < 0.f) {
                hit = true;
                hit_time = time_curr;
                break;
            }
            time_curr = ct;
        }
    }
    __syncwarp();
    if (hit) refine_surface<FMT, STATS>(vol, p, org, dir, hit_time, vx_out, vy_out, vz_out, nx_out, ny_out, nz_out);
    if (inside) {
        const size_t pix = (size_t)W * y + x;
        vmap[3 * pix + 0] = vx_out; vmap[3 * pix + 1] = vy_out; vmap[3 * pix + 2] = vz_out;
        nmap[3 * pix + 0] = nx_out; nmap[3 * pix + 1] = ny_out; nmap[3 * pix + 2] = nz_out;
    }
}

// resize_vertex_map / resize_normal_map (absent from the reference; named at
// common/inc/constants.h:175-176): 2x2 block mean, all four valid.
template <bool NORMAL>
__global__ void resize_map_kernel(const float *src, float *dst, int sc, int sr) {
    const int dc = sc >> 1, dr = sr >> 1;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    allow_next_kernel();
    wait_previous_kernel();
    if (x >= dc || y >= dr) return;
    const float qnan = __int_as_float(0x7fffffff);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    bool ok = true;
    #pragma unroll
    for (int dy = 0; dy < 2; ++dy)
        #pragma unroll
        for (int dx = 0; dx < 2; ++dx) {
            size_t i = 3 * ((size_t)(2 * y + dy) * sc + (2 * x + dx));
            float a = src[i], b = src[i + 1], c = src[i + 2];
            ok = ok && !isnan(a);
            sx = sx + a; sy = sy + b; sz = sz + c;
        }
    float ox = qnan, oy = qnan, oz = qnan;
    if (ok) {
        if (NORMAL) {
            float d = 0.f; d += sx * sx; d += sy * sy; d += sz * sz;
            float rs = 1.f / sqrtf(d);
            ox = sx * rs; oy = sy * rs; oz = sz * rs;
        } else {
            ox = sx * 0.25f; oy = sy * 0.25f; oz = sz * 0.25f;
        }
    }
    size_t o = 3 * ((size_t)y * dc + x);
    dst[o] = ox; dst[o + 1] = oy; dst[o + 2] = oz;
}

// 2x2 mean of a vertex (NORMAL false) or normal map at destination pixel
// (x, y): the same IEEE operations as resize_map_kernel.
template <bool NORMAL>
__device__ __forceinline__ f3 resize_px(const float *__restrict__ src, int sc, int x, int y) {
    const float qnan = __int_as_float(0x7fffffff);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    bool ok = true;
    #pragma unroll
    for (int dy = 0; dy < 2; ++dy)
        #pragma unroll
        for (int dx = 0; dx < 2; ++dx) {
            size_t i = 3 * ((size_t)(2 * y + dy) * sc + (2 * x + dx));
            float a = src[i], b = src[i + 1], c = src[i + 2];
            ok = ok && !isnan(a);
            sx = sx + a; sy = sy + b; sz = sz + c;
        }
    if (!ok) return f3{qnan, qnan, qnan};
    if (NORMAL) {
        float d = 0.f; d += sx * sx; d += sy * sy; d += sz * sz;
        float rs = 1.f / sqrtf(d);
        return f3{sx * rs, sy * rs, sz * rs};
    }
    return f3{sx * 0.25f, sy * 0.25f, sz * 0.25f};
}

// The same mean over four values already in registers (level 1 -> 2).
template <bool NORMAL>
__device__ __forceinline__ f3 mean4(const f3 (&q)[4]) {
    const float qnan = __int_as_float(0x7fffffff);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    bool ok = true;
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        ok = ok && !isnan(q[k].x);
        sx = sx + q[k].x; sy = sy + q[k].y; sz = sz + q[k].z;
    }
    if (!ok) return f3{qnan, qnan, qnan};
    if (NORMAL) {
        float d = 0.f; d += sx * sx; d += sy * sy; d += sz * sz;
        float rs = 1.f / sqrtf(d);
        return f3{sx * rs, sy * rs, sz * rs};
    }
    return f3{sx * 0.25f, sy * 0.25f, sz * 0.25f};
}

__device__ __forceinline__ void put3(float *dst, size_t i, f3 v) {
    dst[3 * i] = v.x; dst[3 * i + 1] = v.y; dst[3 * i + 2] = v.z;
}

// Model-map pyramid in one launch: thread (X, Y) makes level-1 pixels
// (2X..2X+1, 2Y..2Y+1) of the vertex and normal maps and, from those four
// values, level-2 pixel (X, Y) -- the values resize_map_kernel gives level
// by level.  v2/n2 null: level 1 only.
__global__ void resize_model_maps_kernel(const float *__restrict__ v0, const float *__restrict__ n0,
                                         float *__restrict__ v1, float *__restrict__ n1, float *__restrict__ v2,
                                         float *__restrict__ n2, int c0, int r0) {
    const int c1 = c0 >> 1, r1 = r0 >> 1, c2 = c1 >> 1, r2 = r1 >> 1;
    const int X = blockIdx.x * blockDim.x + threadIdx.x;
    const int Y = blockIdx.y * blockDim.y + threadIdx.y;
    if (2 * X >= c1 || 2 * Y >= r1) return;
    f3 qv[4], qn[4];
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = 2 * X + (k & 1), y = 2 * Y + (k >> 1);
        if (x >= c1 || y >= r1) { qv[k] = qn[k] = f3{0.f, 0.f, 0.f}; continue; }
        qv[k] = resize_px<false>(v0, c0, x, y);
        qn[k] = resize_px<true>(n0, c0, x, y);
        put3(v1, (size_t)y * c1 + x, qv[k]);
        put3(n1, (size_t)y * c1 + x, qn[k]);
    }
    if (v2 && X < c2 && Y < r2) {
        put3(v2, (size_t)Y * c2 + X, mean4<false>(qv));
        put3(n2, (size_t)Y * c2 + X, mean4<true>(qn));
    }
}

// transform_map.cl:6-65
__global__ void transform_maps_kernel(const float *__restrict__ vs, const float *__restrict__ ns, float *vd,
                                      float *nd, const tde_matrix3f R, const tde_point3f t, int W, int H) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const float qnan = __int_as_float(0x7fffffff);
    size_t i = 3 * ((size_t)y * W + x);
    f3 v{vs[i], vs[i + 1], vs[i + 2]};
    f3 vo{qnan, qnan, qnan};
    if (!isnan(v.x)) {
        f3 r = mat_vec(R, v);
        vo = f3{r.x + t.x, r.y + t.y, r.z + t.z};
    }
    f3 n{ns[i], ns[i + 1], ns[i + 2]};
    f3 no{qnan, qnan, qnan};
    if (!isnan(n.x)) no = mat_vec(R, n);
    vd[i] = vo.x; vd[i + 1] = vo.y; vd[i + 2] = vo.z;
    nd[i] = no.x; nd[i + 1] = no.y; nd[i + 2] = no.z;
}

}  // namespace

int launch_raycast(const void *volume, int format, float *vmap, float *nmap, const tde_point3f &t,
                   const tde_matrix3f &R, float trunc, const tde_intrinsics &intr, const tde_round_buffer &rb,
                   const tde_point3f &cell, const CamPose *dpose, const uint8_t *neg_flags,
                   const unsigned long long *neg_masks, cudaStream_t stream, bool chained, unsigned *touched) {
    RayParams p;
    p.dpose = dpose;
    p.neg_flags = neg_flags;
    p.t = t; p.R = R;
    p.time_step = (float)((double)trunc * 0.8);
    p.max_time = 3.f * ((rb.volume_size.x + rb.volume_size.y) + rb.volume_size.z);
    p.intr = intr; p.rb = rb; p.cell = cell; p.n = voxel_count(rb);
    p.inv_cell[0] = 1.f / cell.x; p.inv_cell[1] = 1.f / cell.y; p.inv_cell[2] = 1.f / cell.z;
    const bool whole = rb.voxels_size.x % 32 == 0 && rb.voxels_size.y % 32 == 0 && rb.voxels_size.z % 32 == 0;
    p.super_flags = (neg_flags && whole) ? neg_flags + brick_count(rb) : nullptr;
    p.neg_masks = neg_masks;
    p.touched = touched;
    dim3 block(kRayThreads);
    // a grid takes 65,535 blocks of rows; images of more come in layers
    const unsigned row_blocks = div_up(intr.rows, kRayBlockRows), layers = div_up(row_blocks, 65535u);
    dim3 grid(div_up(intr.cols, kRayBlockCols), div_up(row_blocks, layers), layers);
    return dispatch_format(format, [&](auto F) {
        constexpr int FM = decltype(F)::value;
        const auto kernel = [&](auto stats) {
            constexpr bool ST = decltype(stats)::value;
            if (neg_masks)
                return whole ? raycast_kernel<FM, FLAG_MASKS, true, ST> : raycast_kernel<FM, FLAG_MASKS, false, ST>;
            if (neg_flags)
                return whole ? raycast_kernel<FM, FLAG_BYTES, true, ST> : raycast_kernel<FM, FLAG_BYTES, false, ST>;
            return raycast_kernel<FM, FLAG_NONE, false, ST>;
        };
        return launch_chained("raycast", chained, touched ? kernel(std::true_type{}) : kernel(std::false_type{}), grid,
                              block, stream, volume, vmap, nmap, p);
    });
}

int launch_resize_map(const float *src, float *dst, int sc, int sr, bool normal, cudaStream_t stream) {
    dim3 block(32, 8);
    dim3 grid(div_up(sc >> 1, 32), div_up(sr >> 1, 8));
    return launch_chained("resize_map", true, normal ? resize_map_kernel<true> : resize_map_kernel<false>, grid, block,
                          stream, src, dst, sc, sr);
}

int launch_resize_model_maps(const float *v0, const float *n0, float *v1, float *n1, float *v2, float *n2, int c0,
                             int r0, cudaStream_t stream) {
    dim3 block(32, 8);
    dim3 grid(div_up(div_up(c0 >> 1, 2), 32), div_up(div_up(r0 >> 1, 2), 8));
    resize_model_maps_kernel<<<grid, block, 0, stream>>>(v0, n0, v1, n1, v2, n2, c0, r0);
    return check_launch("resize_model_maps");
}

int launch_transform_maps(const float *vs, const float *ns, float *vd, float *nd, const tde_matrix3f &R,
                          const tde_point3f &t, int W, int H, cudaStream_t stream) {
    dim3 block(32, 8);
    dim3 grid(div_up(W, 32), div_up(H, 8));
    transform_maps_kernel<<<grid, block, 0, stream>>>(vs, ns, vd, nd, R, t, W, H);
    return check_launch("transform_maps");
}

}  // namespace tde

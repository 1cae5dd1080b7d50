// The clearance field (vg_check.cuh): per cell of a grid over the workspace, a lower bound of the
// distance from any point of the cell to anything in the environment, so that the checking
// kernels skip the exact queries of spheres that are out of everything's reach.
//
// A cell's bound C is rigorous against the exact tests as they round (collision/sphere_*.hh,
// capt.hh:425-506): no sphere inside the ball of radius C about any point of the cell tests
// negative, neither one about that point nor the members of a larger sphere about it.  The test of
// a primitive or a cloud is negative only if its distance function f at the sphere's centre is
// below the radius, up to a few FP32 roundings; f changes by at most L times the distance moved, so
// f(cell centre) - L * (half the cell's diagonal) - margin bounds it over the cell (and L > 1
// scales it).  The margin is 1 mm + 1e-5 of the coordinates involved, hundreds of times the
// rounding.  min_distance plays no part: a skipped test would have been non-negative, whether or
// not the sorted walk would have reached it.
//
// Built once per change of the environment, when the checks since then make it worth while
// (kFieldStates).  Bound by the distance evaluations (2 M cells x the objects within 0.64 m of
// their 8 x 8 x 8 block).
#include "../../include/vamp_gb300.h"
#include "vg_internal.h"
#include "vg_pool.h"

#include <algorithm>
#include <mutex>

namespace vg
{
    namespace
    {
        constexpr float kCell = 1.0f / kFieldInv;
        constexpr float kCellReach = 0.02166f;   // half of a cell's diagonal, rounded up
        constexpr float kBlockReach = 0.17330f;  // the same of 8 x 8 x 8 cells
        constexpr float kCap = 255.0f / kFieldSteps;
        constexpr int kCells = kFieldCells * kFieldCells * kFieldCells;
        constexpr int kChunk = 1024;  // objects listed at a time
        constexpr int kMaxGap = 27;   // cells; 27 cells are beyond kCap

        __device__ __forceinline__ float len3(float x, float y, float z)
        {
            return sqrtf(fmaf(x, x, fmaf(y, y, z * z)));
        }

        __device__ __forceinline__ float margin(float size)
        {
            return fmaf(1e-5f, size, 1e-3f);
        }

        // A C as above for object o of a kind, over the ball of radius `reach` about (x, y, z):
        // spheres of radius r whose centre is d from there need f >= r, f falls by at most L d, and
        // d + r <= C, so C = (f - L * reach - margin) / max(L, 1).  NaN for objects with non-finite
        // fields.
        __device__ __forceinline__ float object_bound(int kind, const float4 *o, float x, float y, float z, float reach)
        {
            const float4 a = o[0];
            const float place = fabsf(a.x) + fabsf(a.y) + fabsf(a.z) + 4.0f;
            if (kind == 0)
            {
                const float r = fabsf(a.w);
                return len3(x - a.x, y - a.y, z - a.z) - r - reach - margin(place + r);
            }
            const float4 b = o[1];
            if (kind <= 2)
            {
                // the reference tests a point of the segment, whatever rdv holds
                const float vx = kind == 1 ? a.w : 0.0f, vy = kind == 1 ? b.x : 0.0f, vz = b.y;
                const float wx = x - a.x, wy = y - a.y, wz = z - a.z;
                const float vv = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
                float t = vv > 0.0f ? fmaf(wx, vx, fmaf(wy, vy, wz * vz)) / vv : 0.0f;
                t = fminf(fmaxf(t, 0.0f), 1.0f);
                const float r = fabsf(b.z), size = place + r + fabsf(vx) + fabsf(vy) + fabsf(vz);
                return len3(fmaf(-t, vx, wx), fmaf(-t, vy, wy), fmaf(-t, vz, wz)) - r - reach - margin(size);
            }
            // cuboids: f = |max(|A (p - c)| - half extents, 0)| with the axes as rows of A (kind 4
            // reads the horizontal parts of the first two); |A d| <= L |d| with L^2 the largest
            // absolute row sum of A A^T
            const float4 c = o[2], d = o[3];
            const float A[3][3] = {{b.x, b.y, kind == 3 ? b.z : 0.0f},
                                   {c.x, c.y, kind == 3 ? c.z : 0.0f},
                                   {kind == 3 ? d.x : 0.0f, kind == 3 ? d.y : 0.0f, kind == 3 ? d.z : 1.0f}};
            float l2 = 0.0f;
            for (int i = 0; i < 3; ++i)
            {
                float sum = 0.0f;
                for (int j = 0; j < 3; ++j)
                    sum += fabsf(fmaf(A[i][0], A[j][0], fmaf(A[i][1], A[j][1], A[i][2] * A[j][2])));
                l2 = sum > l2 || !(sum == sum) ? sum : l2;
            }
            const float L = sqrtf(l2) * 1.0001f;
            const float h[3] = {a.w, b.w, c.w};
            float e[3];
            for (int i = 0; i < 3; ++i)
            {
                const float v = fabsf(fmaf(A[i][0], x - a.x, fmaf(A[i][1], y - a.y, A[i][2] * (z - a.z)))) - h[i];
                e[i] = v > 0.0f || !(v == v) ? v : 0.0f;
            }
            const float size = (1.0f + L) * place + fabsf(h[0]) + fabsf(h[1]) + fabsf(h[2]);
            return (len3(e[0], e[1], e[2]) - L * reach - margin(size)) / fmaxf(L, 1.0f);
        }

        __device__ __forceinline__ float3 cell_centre(int ix, int iy, int iz)
        {
            return make_float3((static_cast<float>(ix) - kFieldX) * kCell, (static_cast<float>(iy) - kFieldX) * kCell,
                               (static_cast<float>(iz) - kFieldZ) * kCell);
        }

        __device__ __forceinline__ unsigned step_of(float clear)
        {
            return clear > 0.0f ? static_cast<unsigned>(fminf(clear * kFieldSteps, 255.0f)) : 0u;  // NaN: 0
        }

        // Primitives.  A block of threads takes 8 x 8 x 8 cells: the objects that may be within
        // the field's range of the block are listed first (from 60 to a few), then each thread
        // evaluates two cells.
        __global__ void __launch_bounds__(256) field_primitives(const EnvDevice env, uint8_t *out)
        {
            __shared__ unsigned list[kChunk];
            __shared__ int count;
            const int t = threadIdx.x;
            const int bx = blockIdx.x % 16, by = blockIdx.x / 16 % 16, bz = blockIdx.x / 256;
            const float3 bc = cell_centre(8 * bx, 8 * by, 8 * bz);
            const float half = 3.5f * kCell;
            int cell[2];
            float3 p[2];
            float best[2];
            for (int i = 0; i < 2; ++i)
            {
                const int l = t + 256 * i;
                const int ix = 8 * bx + (l & 7), iy = 8 * by + (l >> 3 & 7), iz = 8 * bz + (l >> 6);
                cell[i] = field_at(ix, iy, iz);
                p[i] = cell_centre(ix, iy, iz);
                best[i] = kCap;
            }
            int first[6] = {0, 0, 0, 0, 0, 0};
            for (int k = 0; k < 5; ++k)
                first[k + 1] = first[k] + env.n[k];
            for (int base = 0; base < first[5]; base += kChunk)
            {
                if (t == 0)
                    count = 0;
                __syncthreads();
                for (int i = base + t; i < min(base + kChunk, first[5]); i += 256)
                {
                    int k = 0;
                    while (i >= first[k + 1])
                        ++k;
                    const unsigned at = env.off[k] + (i - first[k]) * rec_f4(k);
                    if (!(object_bound(k, env.buf + at, bc.x + half, bc.y + half, bc.z + half, kBlockReach) > kCap))
                        list[atomicAdd(&count, 1)] = at << 3 | static_cast<unsigned>(k);
                }
                __syncthreads();
                for (int j = 0; j < count; ++j)
                {
                    const int k = list[j] & 7u;
                    const float4 *o = env.buf + (list[j] >> 3);
                    for (int i = 0; i < 2; ++i)
                    {
                        const float b = object_bound(k, o, p[i].x, p[i].y, p[i].z, kCellReach);
                        best[i] = b > 0.0f ? fminf(best[i], b) : 0.0f;
                    }
                }
                __syncthreads();
            }
            for (int i = 0; i < 2; ++i)
                out[cell[i]] = static_cast<uint8_t>(step_of(best[i]));
        }

        // Pointclouds: occupied cells, then the exact squared distance transform of the gaps
        // between cells (per axis max(|i - j| - 1, 0)), one axis at a time.  Points outside the
        // grid count at the nearest cell of its border, which is nearer to every cell inside.
        __device__ __forceinline__ void mark(unsigned *occ, float x, float y, float z)
        {
            if (!(fabsf(x) < 3.4e38f && fabsf(y) < 3.4e38f && fabsf(z) < 3.4e38f))
                return;  // padding and non-finite points are never within reach
            const float top = static_cast<float>(kFieldCells - 1);
            const int ix = static_cast<int>(rintf(fminf(fmaxf(fmaf(x, kFieldInv, kFieldX), 0.0f), top)));
            const int iy = static_cast<int>(rintf(fminf(fmaxf(fmaf(y, kFieldInv, kFieldX), 0.0f), top)));
            const int iz = static_cast<int>(rintf(fminf(fmaxf(fmaf(z, kFieldInv, kFieldZ), 0.0f), top)));
            atomicOr(occ + ((iz << kFieldBits) + iy) * (kFieldCells / 32) + (ix >> 5), 1u << (ix & 31));
        }

        // points [n][3]
        __global__ void field_mark_points(const float *xyz, long long n, unsigned *occ)
        {
            const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i < n)
                mark(occ, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
        }

        // 8-point blocks x[8] y[8] z[8]
        __global__ void field_mark_blocks(const float *aff, long long blocks, unsigned *occ)
        {
            const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i < 8 * blocks)
            {
                const float *b = aff + 24 * (i >> 3) + (i & 7);
                mark(occ, b[0], b[8], b[16]);
            }
        }

        __global__ void __launch_bounds__(kFieldCells) field_gap_x(const unsigned *occ, uint8_t *gx)
        {
            const int i = threadIdx.x;
            const unsigned *row = occ + static_cast<long long>(blockIdx.x) * (kFieldCells / 32);
            int best = kMaxGap + 1;
            int w = i >> 5;
            unsigned m = row[w] & (0xffffffffu >> (31 - (i & 31)));
            while (!m && w > 0)
                m = row[--w];
            if (m)
                best = min(best, i - (32 * w + 31 - __clz(m)));
            w = i >> 5;
            m = row[w] & (0xffffffffu << (i & 31));
            while (!m && w < kFieldCells / 32 - 1)
                m = row[++w];
            if (m)
                best = min(best, 32 * w + __ffs(m) - 1 - i);
            gx[static_cast<long long>(blockIdx.x) * kFieldCells + i] = static_cast<uint8_t>(max(best - 1, 0));
        }

        // The other two axes, four cells in x per thread (one byte or one half word per load took
        // 33 and 39 us), outwards until nothing nearer can come.
        constexpr int kQuads = kFieldCells / 4;
        constexpr int kLines = 8;  // lines of a plane per block

        __global__ void __launch_bounds__(kQuads *kLines) field_gap_y(const uint8_t *gx, uint16_t *gy)
        {
            const int y = static_cast<int>(blockIdx.x) * kLines + threadIdx.y;
            const int plane = static_cast<int>(blockIdx.y) << (2 * kFieldBits);
            const uchar4 *in = reinterpret_cast<const uchar4 *>(gx + plane) + threadIdx.x;
            int best[4] = {kMaxGap * kMaxGap, kMaxGap * kMaxGap, kMaxGap * kMaxGap, kMaxGap * kMaxGap};
            auto take = [&](int row, int g) {
                const uchar4 v = in[row * kQuads];
                best[0] = min(best[0], g + v.x * v.x);
                best[1] = min(best[1], g + v.y * v.y);
                best[2] = min(best[2], g + v.z * v.z);
                best[3] = min(best[3], g + v.w * v.w);
            };
            for (int d = 0; d <= kMaxGap; ++d)
            {
                const int g = max(d - 1, 0) * max(d - 1, 0);
                if (g >= max(max(best[0], best[1]), max(best[2], best[3])))
                    break;
                if (y - d >= 0)
                    take(y - d, g);
                if (y + d < kFieldCells)
                    take(y + d, g);
            }
            reinterpret_cast<ushort4 *>(gy + plane)[y * kQuads + threadIdx.x] =
                make_ushort4(static_cast<uint16_t>(best[0]), static_cast<uint16_t>(best[1]), static_cast<uint16_t>(best[2]),
                             static_cast<uint16_t>(best[3]));
        }

        // the last axis; the field takes the smaller of its value and the clouds' (largest point
        // radius r_point)
        __global__ void __launch_bounds__(kQuads *kLines) field_gap_z(const uint16_t *gy, float r_point, uint8_t *out)
        {
            const int z = blockIdx.y;
            const int at = (static_cast<int>(blockIdx.x) * kLines + threadIdx.y) * kQuads + threadIdx.x;
            constexpr int kPlane = kFieldCells * kQuads;
            const ushort4 *in = reinterpret_cast<const ushort4 *>(gy) + at;
            int best[4] = {kMaxGap * kMaxGap, kMaxGap * kMaxGap, kMaxGap * kMaxGap, kMaxGap * kMaxGap};
            auto take = [&](int plane, int g) {
                const ushort4 v = in[plane * kPlane];
                best[0] = min(best[0], g + v.x);
                best[1] = min(best[1], g + v.y);
                best[2] = min(best[2], g + v.z);
                best[3] = min(best[3], g + v.w);
            };
            for (int d = 0; d <= kMaxGap; ++d)
            {
                const int g = max(d - 1, 0) * max(d - 1, 0);
                if (g >= max(max(best[0], best[1]), max(best[2], best[3])))
                    break;
                if (z - d >= 0)
                    take(z - d, g);
                if (z + d < kFieldCells)
                    take(z + d, g);
            }
            const float less = r_point + margin(r_point + 4.0f);
            auto value = [&](int b, uint8_t have) {
                return static_cast<uint8_t>(min(static_cast<unsigned>(have), step_of(sqrtf(static_cast<float>(b)) * kCell - less)));
            };
            uchar4 *cell = reinterpret_cast<uchar4 *>(out + field_at(4 * threadIdx.x, blockIdx.x * kLines + threadIdx.y, z));
            const uchar4 have = *cell;
            *cell = make_uchar4(value(best[0], have.x), value(best[1], have.y), value(best[2], have.z), value(best[3], have.w));
        }

        // Heightfields (t_heightfield, vg_check.cuh): the test is z - r - z0 < zs * h for the
        // sample of the sphere's own column.  The field also stands for spheres about other
        // centres (a link group's members), so its bound C at p has to keep every sphere inside the
        // ball of radius C about p above the surface: z - z0 - C >= the largest zs * h within C of
        // p, sideways.  Largest zs * h per column of cells first (one more sample on each side,
        // for the rounding of the index), on a grid kMaxGap columns wider than the field; infinity
        // where a field or sample is not finite.
        constexpr int kWide = kFieldCells + 2 * kMaxGap;

        __global__ void field_columns(const HeightView h, float *tops)
        {
            const int ix = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x), iy = blockIdx.y;
            if (ix >= kWide)
                return;
            const float3 p = cell_centre(ix - kMaxGap, iy - kMaxGap, 0);
            const float half = 0.5f * kCell + 1e-4f;
            auto range = [&](float scale, float at, float from, int n, int &lo, int &hi) {
                const float c = fmaf(scale, from - at, static_cast<float>(n / 2)), w = fabsf(scale) * half + 1.0f;
                const float top = static_cast<float>(n);
                lo = static_cast<int>(fminf(fmaxf(c - w, 0.0f), top));
                hi = static_cast<int>(fminf(fmaxf(c + w, 0.0f), top));
            };
            int x0, x1, y0, y1;
            range(h.xs, p.x, h.x, h.xd, x0, x1);
            range(h.ys, p.y, h.y, h.yd, y0, y1);
            const long long last = static_cast<long long>(h.xd) * h.yd - 1;
            bool fine = fabsf(h.x) < 1e3f && fabsf(h.y) < 1e3f && fabsf(h.z) < 1e6f && fabsf(h.xs) < 1e6f && fabsf(h.ys) < 1e6f;
            float top = -3.4e38f;
            for (int y = y0; y <= y1 && fine; ++y)
            {
                for (int x = x0; x <= x1; ++x)
                {
                    const long long i = static_cast<long long>(y) * h.xd + x;
                    const float v = h.zs * h.data[i < last ? i : last];
                    fine = fine && fabsf(v) < 1e6f;  // false for NaN
                    top = fmaxf(top, v);
                }
            }
            tops[iy * kWide + ix] = fine ? top : __int_as_float(0x7f800000);
        }

        // A window of R columns to each side holds everything within (R - 1) cells of the middle
        // column's points: C is the best of min((R - 1) cells, z - z0 - the window's largest) over
        // a few R.
        __global__ void __launch_bounds__(kFieldCells) field_heights(const HeightView h, const float *tops, uint8_t *out)
        {
            constexpr int kRings = 5;
            constexpr int kWindow[kRings] = {2, 4, 8, 16, kMaxGap};
            const int ix = threadIdx.x, iy = blockIdx.x;
            float top[kRings];
            float best = -3.4e38f;
            int done = -1;
#pragma unroll
            for (int r = 0; r < kRings; ++r)
            {
                for (int dy = -kWindow[r]; dy <= kWindow[r]; ++dy)
                {
                    const float *row = tops + (iy + kMaxGap + dy) * kWide + ix + kMaxGap;
                    const bool inner = dy >= -done && dy <= done;
                    for (int dx = -kWindow[r]; dx <= kWindow[r]; ++dx)
                    {
                        if (inner && dx == -done)
                            dx = done + 1;  // columns of the window before
                        best = fmaxf(best, row[dx]);
                    }
                }
                done = kWindow[r];
                top[r] = best;
            }
            for (int iz = 0; iz < kFieldCells; ++iz)
            {
                uint8_t *cell = out + field_at(ix, iy, iz);
                const float z = (static_cast<float>(iz) - kFieldZ) * kCell;
                float clear = 0.0f;
#pragma unroll
                for (int r = 0; r < kRings; ++r)
                {
                    const float up = z - h.z - top[r] - 0.5f * kCell - margin(8.0f + fabsf(h.z) + fabsf(top[r]));
                    clear = fmaxf(clear, fminf(static_cast<float>(kWindow[r] - 1) * kCell - margin(8.0f), up));
                }
                *cell = static_cast<uint8_t>(min(static_cast<unsigned>(*cell), step_of(clear)));
            }
        }

        // launches that fill e->d_field on stream s (scratch behind it: occupancy bits and gaps of the
        // clouds, then a heightfield's columns)
        constexpr size_t kScratch = kCells / 8 + 3 * static_cast<size_t>(kCells);
        static_assert(kScratch >= kWide * kWide * sizeof(float), "a heightfield's columns fit the scratch");

        cudaError_t launch_build(vg_env *e, cudaStream_t s)
        {
            unsigned char *scratch = e->d_field + kCells;
            field_primitives<<<kCells / 512, 256, 0, s>>>(env_device(e, nullptr), e->d_field);
            cudaError_t err = cudaGetLastError();
            if (!e->clouds.empty() && err == cudaSuccess)
            {
                unsigned *occ = reinterpret_cast<unsigned *>(scratch);
                uint8_t *gx = scratch + kCells / 8;
                uint16_t *gy = reinterpret_cast<uint16_t *>(gx + kCells);
                float r_point = 0.0f;
                err = cudaMemsetAsync(occ, 0, kCells / 8, s);
                for (size_t i = 0; i < e->clouds.size() && err == cudaSuccess; ++i)
                {
                    const CaptHost &c = e->clouds[i];
                    r_point = std::max(r_point, c.r_point);
                    const CloudPoints &p = e->d_points[i];
                    const long long n = static_cast<long long>(p.n ? p.n : 8 * c.blocks());
                    if (n == 0)
                        continue;
                    const unsigned grid = static_cast<unsigned>((n + 255) / 256);
                    if (p.n)
                        field_mark_points<<<grid, 256, 0, s>>>(p.d, n, occ);
                    else
                        field_mark_blocks<<<grid, 256, 0, s>>>(e->capt_q[i].aff_q, n / 8, occ);
                    err = cudaGetLastError();
                }
                if (err == cudaSuccess)
                {
                    field_gap_x<<<kFieldCells * kFieldCells, kFieldCells, 0, s>>>(occ, gx);
                    const dim3 lines(kQuads, kLines), planes(kFieldCells / kLines, kFieldCells);
                    field_gap_y<<<planes, lines, 0, s>>>(gx, gy);
                    field_gap_z<<<planes, lines, 0, s>>>(gy, r_point, e->d_field);
                    err = cudaGetLastError();
                }
            }
            for (size_t i = 0; i < e->hf.size() && err == cudaSuccess; ++i)
            {
                HeightView h = e->hf[i];
                h.data = static_cast<const float *>(e->d_hf[i]);
                float *tops = reinterpret_cast<float *>(scratch);
                field_columns<<<dim3((kWide + 127) / 128, kWide), 128, 0, s>>>(h, tops);
                field_heights<<<kFieldCells, kFieldCells, 0, s>>>(h, tops, e->d_field);
                err = cudaGetLastError();
            }
            return err;
        }
    }  // namespace

    namespace
    {
        // This thread's calls do not count as unsafe for another thread's capture (in the default, global
        // mode, an allocation or an event's query anywhere would end it).
        struct OutsideCaptures
        {
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;

            OutsideCaptures()
            {
                cudaThreadExchangeStreamCaptureMode(&mode);
            }

            ~OutsideCaptures()
            {
                cudaThreadExchangeStreamCaptureMode(&mode);
            }
        };

        bool captured(cudaStream_t s)
        {
            cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
            if (cudaStreamIsCapturing(s, &status) != cudaSuccess)
            {
                cudaGetLastError();
                return true;
            }
            return status != cudaStreamCaptureStatusNone;
        }
    }  // namespace

    void release_field(vg_env *e)
    {
        pool_give(e->d_field, 0);
        e->d_field = nullptr;
        if (e->field_built)
            cudaEventDestroy(e->field_built);
        e->field_built = nullptr;
    }

    void want_field(vg_env *e, double states, cudaStream_t s)
    {
        if (e->field_ready.load(std::memory_order_acquire))
        {
            return;
        }
        std::lock_guard<std::mutex> lock(e->field_mu);
        e->field_states += states;
        if (e->field_ready.load(std::memory_order_relaxed) || e->field_states < kFieldStates)
        {
            return;
        }
        // the build belongs to no graph: launches under capture run without the field
        if (captured(s))
        {
            return;
        }
        const OutsideCaptures outside;
        cudaError_t err = cudaSuccess;
        if (!e->field_built)
            err = cudaEventCreateWithFlags(&e->field_built, cudaEventDisableTiming);
        if (err == cudaSuccess && !e->d_field)
            err = pool_take(reinterpret_cast<void **>(&e->d_field), kCells + kScratch, s);
        if (err == cudaSuccess)
            err = launch_build(e, s);
        // the call waits for nothing: checks on other streams queue behind this (usable_field)
        if (err == cudaSuccess)
            err = cudaEventRecord(e->field_built, s);
        if (err != cudaSuccess)
        {
            // without a field the checks are as they were; not tried again before the next change
            cudaGetLastError();
            e->field_states = -1e300;
            return;
        }
        e->field_done.store(false, std::memory_order_relaxed);
        ++e->version;  // graphs captured without the field are captured again
        e->field_ready.store(true, std::memory_order_release);
    }

    const uint8_t *usable_field(const vg_env *e, cudaStream_t s)
    {
        if (!e->field_ready.load(std::memory_order_acquire))
        {
            return nullptr;
        }
        if (e->field_done.load(std::memory_order_acquire))
        {
            return e->d_field;
        }
        const OutsideCaptures outside;
        if (cudaEventQuery(e->field_built) == cudaSuccess)
        {
            e->field_done.store(true, std::memory_order_release);
            return e->d_field;
        }
        cudaGetLastError();  // not ready
        // a graph cannot wait for the build
        if (captured(s) || cudaStreamWaitEvent(s, e->field_built, 0) != cudaSuccess)
        {
            cudaGetLastError();
            return nullptr;
        }
        return e->d_field;
    }
}  // namespace vg

// deposit.cu -- species sort, kernel deposit (DENSITY), RENORM_DENSITY and
// the true-TSC deposit (INTERPOLATE_DENSITY_TSC) on sm_100a.
//
// Accumulation: every cloud term keeps the reference's REAL*4 expression
// (BAS*W(i)*W(j)*W(k), left to right).  Terms are summed in float64 and
// rounded once to float32, so the result depends on the particle order only
// through float64 rounding, unlike the reference's REDUCTION(+:U1)
// (grids.f:787-791) whose float32 sum does.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/reverse_iterator.h>

#include "common.cuh"

#define KW (2 * ASOHF_NMAX_KERNELS + 1)

// ------------------------------------------------------------ host tables
// One level of COMPUTE_KERNELS (grids.f:997-1067), host side, same REAL*4
// arithmetic; kk points at W(0).
static void compute_kernel_level(int ir, int deg, float* kk) {
  int n = 1 << ir;
  float h32 = (float)n + 0.5f;
  float h = 2.0f * h32 / 3.0f;
  for (int i = -n; i <= n; i++) {
    if (deg == 2) {
      float bas = (float)abs(i) / h;
      if (bas <= 0.5f) {
        kk[i] = 0.75f - bas * bas;
      } else {
        float t = 1.5f - bas;
        kk[i] = 0.5f * (t * t);
      }
    } else {
      float bas = (float)abs(i) / h32;
      kk[i] = 1.0f - bas;
    }
  }
  float bas = 0.0f;
  for (int i = -n; i <= n; i++)
    for (int j = -n; j <= n; j++)
      for (int q = -n; q <= n; q++) {
        volatile float t = kk[i] * kk[j];  // keep two roundings on the host too
        t = t * kk[q];
        bas = bas + t;
      }
  bas = 1.0f / powf(bas, 1.0f / 3.0f);
  for (int i = -n; i <= n; i++) kk[i] = bas * kk[i];
}

// The tables of levels 0 .. nl, host and device, (NLEVELS+1) rows of KW kept by
// the context: they depend on nothing but the degree, and the sequential sum of
// a level's (2^(l+1)+1)^3 terms takes the host 1.5 ms to level 6.
static int kernel_tables(asohf_ctx* c, int nl, int deg, const float** hk, float** dk) {
  const int d = deg - 1;
  const size_t bytes = sizeof(float) * KW * (ASOHF_NLEVELS + 1);
  if (!c->h_kern[d]) {
    c->h_kern[d] = (float*)calloc(1, bytes);
    if (!c->h_kern[d]) return ASOHF_ERR_CAPACITY;
  }
  if (!c->d_kern[d]) ASOHF_CUDA(cudaMalloc(&c->d_kern[d], bytes));
  const int l0 = c->kern_nl[d] + 1;
  if (l0 <= nl) {
    float* row = c->h_kern[d] + (size_t)l0 * KW;
    for (int ir = l0; ir <= nl; ir++) compute_kernel_level(ir, deg, c->h_kern[d] + (size_t)ir * KW + ASOHF_NMAX_KERNELS);
    ASOHF_CHECK(upload_table(c, c->d_kern[d] + (size_t)l0 * KW, row, sizeof(float) * KW * (size_t)(nl - l0 + 1)));
    c->kern_nl[d] = nl;
  }
  *hk = c->h_kern[d];
  *dk = c->d_kern[d];
  return ASOHF_OK;
}

// ------------------------------------------------------------ species sort
__device__ __forceinline__ int ngp_index(float v, float xmin, float dx, int nx) {
  int i = (int)((v - xmin) / dx) + 1;
  if (i < 1) i = 1;
  if (i > nx) i = nx;
  return i - 1;
}

__global__ void k_ngp_count(const float* __restrict__ x, const float* __restrict__ y,
                            const float* __restrict__ z, int64_t n, int nx, float dx, float xmin,
                            int32_t* __restrict__ cell, int32_t* __restrict__ counts) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int ix = ngp_index(x[i], xmin, dx, nx), jy = ngp_index(y[i], xmin, dx, nx),
        kz = ngp_index(z[i], xmin, dx, nx);
    int c = (kz * nx + jy) * nx + ix;
    cell[i] = c;
    atomicAdd(&counts[c], 1);
  }
}

// dens(cell) for equal masses: the float32 running sum of `count` copies of
// m, as the sequential loop of reader.f:190-201 produces it, divided by bas.
__global__ void k_cell_density_eqmass(const int32_t* __restrict__ counts, int64_t g, float m,
                                      float bas, float* __restrict__ dens) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g;
       c += (int64_t)gridDim.x * blockDim.x) {
    int k = counts[c];
    float s = 0.0f;
    for (int q = 0; q < k; q++) s = __fadd_rn(s, m);
    dens[c] = s / bas;
  }
}

// General masses: the particles of a cell in input order (stable sort), one
// chain of REAL*4 additions a cell.  A thread takes a cell of up to
// CELL_SERIAL particles; the others go to a list that k_cell_density_heavy
// takes by warps, which fetch 32 masses at a time and run the chain on
// broadcasts (in a thread each link waited for two dependent loads: 1.4M
// particles with the sort 0.95 ms, so 0.38).
#define CELL_SERIAL 32
__global__ void k_cell_density_general(const int32_t* __restrict__ offs, const int32_t* __restrict__ order,
                                       const float* __restrict__ m, int64_t g, float bas,
                                       float* __restrict__ dens, int32_t* __restrict__ heavy,
                                       int32_t* __restrict__ nheavy) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int a = offs[c], b = offs[c + 1];
    if (b - a > CELL_SERIAL) {
      heavy[atomicAdd(nheavy, 1)] = (int32_t)c;
      continue;
    }
    float s = 0.0f;
    for (int q = a; q < b; q++) s = __fadd_rn(s, m[order[q]]);
    dens[c] = s / bas;
  }
}

__global__ void k_cell_density_heavy(const int32_t* __restrict__ offs, const int32_t* __restrict__ order,
                                     const float* __restrict__ m, float bas, const int32_t* __restrict__ heavy,
                                     const int32_t* __restrict__ nheavy, float* __restrict__ dens) {
  const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5, n = *nheavy;
  for (int h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; h < n; h += nw) {
    const int c = heavy[h], a = offs[c], b = offs[c + 1];
    float s = 0.0f;
    float v = a + lane < b ? m[order[a + lane]] : 0.0f;
    for (int q = a; q < b; q += 32) {
      const float next = q + 32 + lane < b ? m[order[q + 32 + lane]] : 0.0f;  // in flight during the chain
      if (b - q >= 32) {
#pragma unroll
        for (int l = 0; l < 32; l++) s = __fadd_rn(s, __shfl_sync(0xffffffffu, v, l));
      } else {
        for (int l = 0; l < b - q; l++) s = __fadd_rn(s, __shfl_sync(0xffffffffu, v, l));
      }
      v = next;
    }
    if (lane == 0) dens[c] = s / bas;
  }
}

__global__ void k_species(const int32_t* __restrict__ cell, const float* __restrict__ dens,
                          int64_t n, int n_esp, float log8, uint8_t* __restrict__ spec) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float b = dens[cell[i]];
    int l = 0;
    if (b > 0.0f) {
      // LOG of a REAL*4 rounded to float32 (correctly rounded), then the
      // REAL*4 quotient by LOG(8.0) and INT truncation.
      float lb = (float)log((double)b);
      l = (int)(lb / log8);
      if (l > n_esp - 1) l = n_esp - 1;
      if (l < 0) l = 0;
    }
    spec[i] = (uint8_t)l;
  }
}

#define SPEC_CHUNK 4096
#define SPEC_BLOCK 256

__global__ void k_species_block_counts(const uint8_t* __restrict__ spec, int64_t n, int nb,
                                       int32_t* __restrict__ bc) {
  __shared__ int cnt[ASOHF_N_ESP];
  if (threadIdx.x < ASOHF_N_ESP) cnt[threadIdx.x] = 0;
  __syncthreads();
  int64_t lo = (int64_t)blockIdx.x * SPEC_CHUNK, hi = min(lo + SPEC_CHUNK, n);
  for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) atomicAdd(&cnt[spec[i]], 1);
  __syncthreads();
  if (threadIdx.x < ASOHF_N_ESP) bc[(int64_t)threadIdx.x * nb + blockIdx.x] = cnt[threadIdx.x];
}

// Stable scatter of the store itself: particle i of a block goes to
// offset(species, block) + its rank in the block, its fields and its row in one
// go.  Particles of one species keep their order, so a warp reads the eight
// arrays in order and writes a short run for each species it holds: 32 bytes
// read and 64 written a particle.  56.6M particles: 1.8 ms; 2.5 ms as a
// permutation array, a row copy of the store and a gather of its rows.
__global__ void __launch_bounds__(SPEC_BLOCK)
k_species_scatter(const uint8_t* __restrict__ spec, int64_t n, int nb, const int32_t* __restrict__ boff,
                  DevParticles src, DevParticles dst, float4* __restrict__ rows) {
  __shared__ int wcnt[SPEC_BLOCK / 32][ASOHF_N_ESP];
  __shared__ int run[ASOHF_N_ESP];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x < ASOHF_N_ESP) run[threadIdx.x] = boff[(int64_t)threadIdx.x * nb + blockIdx.x];
  __syncthreads();
  int64_t lo = (int64_t)blockIdx.x * SPEC_CHUNK, hi = min(lo + SPEC_CHUNK, n);
  for (int64_t base = lo; base < hi; base += SPEC_BLOCK) {
    int64_t i = base + threadIdx.x;
    int s = -1;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (i < hi) {
      s = spec[i];
      a = make_float4(src.x[i], src.y[i], src.z[i], src.m[i]);
      b = make_float4(src.vx[i], src.vy[i], src.vz[i], __int_as_float(src.id[i]));
    }
    // rank among the warp's particles of the same species
    const unsigned same = __match_any_sync(0xffffffffu, s);
    const int myrank = __popc(same & ((1u << lane) - 1));
    if (lane < ASOHF_N_ESP) wcnt[wid][lane] = 0;
    __syncwarp();
    if (s >= 0 && myrank == 0) wcnt[wid][s] = __popc(same);
    __syncthreads();
    if (s >= 0) {
      int off = run[s];
      for (int w = 0; w < wid; w++) off += wcnt[w][s];
      const int64_t d = off + myrank;
      dst.x[d] = a.x; dst.y[d] = a.y; dst.z[d] = a.z; dst.m[d] = a.w;
      dst.vx[d] = b.x; dst.vy[d] = b.y; dst.vz[d] = b.z; dst.id[d] = __float_as_int(b.w);
      rows[2 * d] = a;
      rows[2 * d + 1] = b;
    }
    __syncthreads();
    if (threadIdx.x < ASOHF_N_ESP) {
      int t = 0;
      for (int w = 0; w < SPEC_BLOCK / 32; w++) t += wcnt[w][threadIdx.x];
      run[threadIdx.x] += t;
    }
    __syncthreads();
  }
}

// Store permutation in two passes: the store is packed row-wise (one
// 32-byte row per particle, read and written in order), then each output
// particle reads its whole source row with one random 32-byte access; a
// gather straight from the eight arrays would touch eight sectors per
// particle.
__global__ void k_pack_rows(int64_t n, DevParticles s, float4* __restrict__ rows) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    rows[2 * i] = make_float4(s.x[i], s.y[i], s.z[i], s.m[i]);
    rows[2 * i + 1] = make_float4(s.vx[i], s.vy[i], s.vz[i], __int_as_float(s.id[i]));
  }
}

// New store (fields and rows) in the order perm gives: d[i] = old[perm[i]].
// Four particles per thread and step: their rows are all requested before
// any is written.
__global__ void k_gather_rows(const int64_t* __restrict__ perm, int64_t n, const float4* __restrict__ rows,
                              DevParticles d, float4* __restrict__ out_rows) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
    int64_t j[4];
    float4 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int64_t i = i0 + u * stride;
      j[u] = i < n ? perm[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * stride < n) {
        a[u] = rows[2 * j[u]];
        b[u] = rows[2 * j[u] + 1];
      }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int64_t i = i0 + u * stride;
      if (i < n) {
        d.x[i] = a[u].x; d.y[i] = a[u].y; d.z[i] = a[u].z; d.m[i] = a[u].w;
        d.vx[i] = b[u].x; d.vy[i] = b[u].y; d.vz[i] = b[u].z; d.id[i] = __float_as_int(b[u].w);
        out_rows[2 * i] = a[u];
        out_rows[2 * i + 1] = b[u];
      }
    }
  }
}

__global__ void k_iota(int32_t* __restrict__ a, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    a[i] = (int32_t)i;
}

// Room for the row copies of n particles.
static int rows_reserve(asohf_ctx* c, int64_t n) {
  if (c->rows_cap < n) {
    ASOHF_CUDA(cudaStreamSynchronize(c->stream));
    cudaFree(c->rows[0]);
    cudaFree(c->rows[1]);
    c->rows[0] = c->rows[1] = nullptr;
    c->rows_cap = 0;
    c->rows_cur = -1;
    ASOHF_CUDA(cudaMalloc(&c->rows[0], 32 * (size_t)(n > 0 ? n : 1)));
    ASOHF_CUDA(cudaMalloc(&c->rows[1], 32 * (size_t)(n > 0 ? n : 1)));
    c->rows_cap = n;
  }
  return ASOHF_OK;
}

int permute_store(asohf_ctx* c, const int64_t* perm) {
  int64_t n = c->p.n;
  ASOHF_CHECK(rows_reserve(c, n));
  {
    int kt_ = ktime_begin(c, "store_permute");
    int src = c->rows_cur;
    if (src < 0) {  // no row copy of the current order yet
      src = 0;
      k_pack_rows<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(n, c->p, c->rows[0]);
      c->launches++;
    }
    k_gather_rows<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(perm, n, c->rows[src], c->alt,
                                                                          c->rows[1 - src]);
    c->rows_cur = 1 - src;
    ktime_end(c, kt_);
  }
  c->launches++;
  ASOHF_CUDA(cudaGetLastError());
  ctx_swap_particles(c);
  return ASOHF_OK;
}

extern "C" int asohf_sort_dm_particles_localdensity(asohf_ctx* c, int nx, float dx, float rodo,
                                                    float re0, int32_t* npart_esp) {
  if (!c || nx <= 0 || !npart_esp) return ASOHF_ERR_INVALID;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  int64_t n = c->p.n;
  int64_t g = (int64_t)nx * nx * nx;
  int nb = (int)((n + SPEC_CHUNK - 1) / SPEC_CHUNK);
  if (nb < 1) nb = 1;
  bool eq = (c->mmin == c->norma);
  size_t cub_bytes = 0;
  int cell_bits = 1;
  if (!eq) {
    while ((1ll << cell_bits) < g) cell_bits++;
    cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, (int32_t*)nullptr, (int32_t*)nullptr,
                                    (int32_t*)nullptr, (int32_t*)nullptr, (int)n, 0, cell_bits);
  }
  size_t cub_scan = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, cub_scan, (int32_t*)nullptr, (int32_t*)nullptr,
                                (int)(nb * ASOHF_N_ESP));
  size_t cub_scan2 = 0;
  if (!eq) cub::DeviceScan::ExclusiveSum(nullptr, cub_scan2, (int32_t*)nullptr, (int32_t*)nullptr, (int)(g + 1));
  size_t need = 4 * n + 4 * g + 4 * g + n + 4 * (size_t)nb * ASOHF_N_ESP * 2 +
                (eq ? 0 : (16 * n + n / 8 + 4 * (g + 1) * 2 + cub_bytes + cub_scan2)) + cub_scan + 8192;
  ASOHF_CHECK(arena_reserve(c, need));
  int32_t* cell = (int32_t*)arena_alloc(c, 4 * n);
  int32_t* counts = (int32_t*)arena_alloc(c, 4 * g);
  float* dens = (float*)arena_alloc(c, 4 * g);
  uint8_t* spec = (uint8_t*)arena_alloc(c, n + 16);
  int32_t* bc = (int32_t*)arena_alloc(c, 4 * (size_t)nb * ASOHF_N_ESP);
  int32_t* boff = (int32_t*)arena_alloc(c, 4 * (size_t)nb * ASOHF_N_ESP);
  void* tscan = arena_alloc(c, cub_scan);
  ASOHF_CUDA(cudaMemsetAsync(counts, 0, 4 * g, c->stream));
  float xmin = -((float)nx * dx) / 2.0f;
  {
    int kt_ = ktime_begin(c, "species_ngp_count");
    k_ngp_count<<<grid_for(n, 256), 256, 0, c->stream>>>(c->p.x, c->p.y, c->p.z, n, nx, dx, xmin,
                                                       cell, counts);
    ktime_end(c, kt_);
  }
  c->launches++;
  float bas = dx * dx * dx * rodo * (re0 * re0 * re0);
  if (eq) {
    {
      int kt_ = ktime_begin(c, "species_cell_density");
      k_cell_density_eqmass<<<grid_for(g, 256), 256, 0, c->stream>>>(counts, g, c->norma, bas, dens);
      ktime_end(c, kt_);
    }
    c->launches++;
  } else {
    // particles of each cell in input order: stable radix sort of (cell, i)
    int32_t* idx = (int32_t*)arena_alloc(c, 4 * n);
    int32_t* cell_s = (int32_t*)arena_alloc(c, 4 * n);
    int32_t* order = (int32_t*)arena_alloc(c, 4 * n);
    int32_t* offs = (int32_t*)arena_alloc(c, 4 * (g + 1));
    int32_t* cnt1 = (int32_t*)arena_alloc(c, 4 * (g + 1));
    void* tsort = arena_alloc(c, cub_bytes);
    void* tscan2 = arena_alloc(c, cub_scan2);
    int32_t* heavy = (int32_t*)arena_alloc(c, 4 * (n / CELL_SERIAL + 1));
    int32_t* nheavy = (int32_t*)arena_alloc(c, 4);
    if (!idx || !cell_s || !order || !offs || !cnt1 || !tsort || !tscan2 || !heavy || !nheavy) return ASOHF_ERR_CAPACITY;
    int kt_ = ktime_begin(c, "species_cell_density");
    k_iota<<<grid_for(n, 256), 256, 0, c->stream>>>(idx, n);
    ASOHF_CUDA(cub::DeviceRadixSort::SortPairs(tsort, cub_bytes, cell, cell_s, idx, order, (int)n, 0,
                                               cell_bits, c->stream));
    ASOHF_CUDA(cudaMemsetAsync(cnt1 + g, 0, 4, c->stream));
    ASOHF_CUDA(cudaMemcpyAsync(cnt1, counts, 4 * g, cudaMemcpyDeviceToDevice, c->stream));
    ASOHF_CUDA(cub::DeviceScan::ExclusiveSum(tscan2, cub_scan2, cnt1, offs, (int)(g + 1), c->stream));
    ASOHF_CUDA(cudaMemsetAsync(nheavy, 0, 4, c->stream));
    k_cell_density_general<<<grid_for(g, 256), 256, 0, c->stream>>>(offs, order, c->p.m, g, bas, dens, heavy, nheavy);
    k_cell_density_heavy<<<c->num_sms * 4, 256, 0, c->stream>>>(offs, order, c->p.m, bas, heavy, nheavy, dens);
    ktime_end(c, kt_);
    c->launches += 3;
  }
  {
    int kt_ = ktime_begin(c, "species_classify");
    k_species<<<grid_for(n, 256), 256, 0, c->stream>>>(cell, dens, n, ASOHF_N_ESP, logf(8.0f), spec);
    k_species_block_counts<<<nb, SPEC_BLOCK, 0, c->stream>>>(spec, n, nb, bc);
    ASOHF_CUDA(cub::DeviceScan::ExclusiveSum(tscan, cub_scan, bc, boff, nb * ASOHF_N_ESP, c->stream));
    ktime_end(c, kt_);
  }
  ASOHF_CHECK(rows_reserve(c, n));
  {
    int kt_ = ktime_begin(c, "species_scatter");
    const int to = c->rows_cur == 0 ? 1 : 0;
    k_species_scatter<<<nb, SPEC_BLOCK, 0, c->stream>>>(spec, n, nb, boff, c->p, c->alt, c->rows[to]);
    c->rows_cur = to;
    ktime_end(c, kt_);
  }
  c->launches += 4;
  ASOHF_CUDA(cudaGetLastError());
  ctx_swap_particles(c);
  // the last block's offset and count of each species (strided copies)
  int32_t tot[ASOHF_N_ESP];
  int32_t last_off[ASOHF_N_ESP], last_cnt[ASOHF_N_ESP];
  ASOHF_CUDA(cudaMemcpy2DAsync(last_off, 4, boff + nb - 1, 4 * (size_t)nb, 4, ASOHF_N_ESP, cudaMemcpyDeviceToHost,
                               c->stream));
  ASOHF_CUDA(cudaMemcpy2DAsync(last_cnt, 4, bc + nb - 1, 4 * (size_t)nb, 4, ASOHF_N_ESP, cudaMemcpyDeviceToHost,
                               c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  int64_t prev = 0;
  for (int s = 0; s < ASOHF_N_ESP; s++) {
    int64_t end = (int64_t)last_off[s] + last_cnt[s];
    tot[s] = (int32_t)(end - prev);
    prev = end;
  }
  if (prev != n) return ASOHF_ERR_WRONG_SORTING;
  memcpy(npart_esp, tot, sizeof(tot));
  return ASOHF_OK;
}

// ------------------------------------------------------------ base deposit
// The 27-cell periodic cloud of grids.f:787-820 for particles whose host
// cell lies in the box; BASE_OUTLIER handles the rest (positions more than
// one cell outside the box), with the same wrap-once arithmetic.
__device__ __forceinline__ int wrap_once(int i, int nx) {
  if (i > nx) i -= nx;
  if (i < 1) i += nx;
  return i;
}

// One particle's cloud by float64 atomics.
__device__ __forceinline__ void base_cloud(int ix, int jy, int kz, float bas, const float* w, int nx,
                                           double* __restrict__ acc) {
  for (int kk = -1; kk <= 1; kk++)
    for (int jj = -1; jj <= 1; jj++)
      for (int ii = -1; ii <= 1; ii++) {
        int i1 = wrap_once(ix + ii, nx), j1 = wrap_once(jy + jj, nx), k1 = wrap_once(kz + kk, nx);
        if (i1 < 1 || i1 > nx || j1 < 1 || j1 > nx || k1 < 1 || k1 > nx) continue;  // outside the box
        float t = __fmul_rn(__fmul_rn(__fmul_rn(bas, w[ii + 1]), w[jj + 1]), w[kk + 1]);
        atomicAdd(&acc[((size_t)(k1 - 1) * nx + (j1 - 1)) * nx + (i1 - 1)], (double)t);
      }
}

// Particles whose host cell lies outside the box, when the counts met any,
// summed into the float64 grid the stencil then left.
__global__ void k_density_base_outliers(const float* __restrict__ x, const float* __restrict__ y,
                                        const float* __restrict__ z, const float* __restrict__ m, int64_t n,
                                        int nx, float xl, float dx, const float* __restrict__ k0,
                                        const int* __restrict__ outside, double* __restrict__ acc) {
  if (!*outside) return;
  float w[3] = {k0[0], k0[1], k0[2]};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)((x[i] - xl) / dx) + 1;
    int jy = (int)((y[i] - xl) / dx) + 1;
    int kz = (int)((z[i] - xl) / dx) + 1;
    if (ix >= 1 && ix <= nx && jy >= 1 && jy <= nx && kz >= 1 && kz <= nx) continue;
    base_cloud(ix, jy, kz, m[i], w, nx, acc);
  }
}

// Every particle with global float64 atomics, in store order (no patches, so
// no binned copy).
__global__ void k_density_base_all(const float* __restrict__ x, const float* __restrict__ y,
                                   const float* __restrict__ z, const float* __restrict__ m, int64_t n, int nx,
                                   float xl, float dx, const float* __restrict__ k0, double* __restrict__ acc) {
  float w[3] = {k0[0], k0[1], k0[2]};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)((x[i] - xl) / dx) + 1;
    int jy = (int)((y[i] - xl) / dx) + 1;
    int kz = (int)((z[i] - xl) / dx) + 1;
    base_cloud(ix, jy, kz, m[i], w, nx, acc);
  }
}

// The binned copy, whose order keeps a cell's particles together: a warp takes
// 32 of them and deposits one run of equal host cells at a time, lane t < 27 on
// target t: the run's terms are summed first, then one atomic a target.  1.4M
// particles of two masses on 96^3 in 0.09 ms; 0.59 ms with an atomic a term in
// store order, which met on the cells of halo cores.
__global__ void k_density_base_runs(const float4* __restrict__ P, const uint8_t* __restrict__ S, int64_t n, int nx,
                                    float xl, float dx, const float* __restrict__ k0, double* __restrict__ acc) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i3 = lane % 3, j3 = (lane / 3) % 3, k3 = min(lane / 9, 2);
  const float wi = k0[i3], wj = k0[j3], wk = k0[k3];
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n; base += nw * 32) {
    const int64_t q = base + lane;
    const bool live = q < n && S[q] != 255;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) p = P[q];
    const int ix = (int)((p.x - xl) / dx) + 1, jy = (int)((p.y - xl) / dx) + 1, kz = (int)((p.z - xl) / dx) + 1;
    const int pi = __shfl_up_sync(FULL, ix, 1), pj = __shfl_up_sync(FULL, jy, 1), pk = __shfl_up_sync(FULL, kz, 1);
    const int pl = __shfl_up_sync(FULL, live ? 1 : 0, 1);
    unsigned heads = __ballot_sync(FULL, live && (lane == 0 || !pl || pi != ix || pj != jy || pk != kz));
    const unsigned alive = __ballot_sync(FULL, live);
    while (heads) {
      const int a = __ffs(heads) - 1;
      heads &= heads - 1;
      // the run: live lanes from a to the next head or the first dead lane
      unsigned grp = FULL << a;
      if (heads) grp &= (1u << (__ffs(heads) - 1)) - 1u;
      const unsigned dead = ~alive & grp;
      if (dead) grp &= (1u << (__ffs(dead) - 1)) - 1u;
      const int e = 32 - __clz(grp);
      double s = 0.0;
      for (int l = a; l < e; l++) {
        const float m = __shfl_sync(FULL, p.w, l);
        s += (double)__fmul_rn(__fmul_rn(__fmul_rn(m, wi), wj), wk);
      }
      const int i1 = wrap_once(__shfl_sync(FULL, ix, a) + i3 - 1, nx),
                j1 = wrap_once(__shfl_sync(FULL, jy, a) + j3 - 1, nx),
                k1 = wrap_once(__shfl_sync(FULL, kz, a) + k3 - 1, nx);
      if (lane < 27 && i1 >= 1 && i1 <= nx && j1 >= 1 && j1 <= nx && k1 >= 1 && k1 <= nx)
        atomicAdd(&acc[((size_t)(k1 - 1) * nx + (j1 - 1)) * nx + (i1 - 1)], s);
    }
  }
}

// u1 of a grid whose stencil found particles outside the box (else it wrote u1
// itself).
__global__ void k_finish_outliers(const int* __restrict__ outside, const double* __restrict__ acc, int64_t g,
                                  float denbas, float* __restrict__ u1) {
  if (!*outside) return;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g;
       c += (int64_t)gridDim.x * blockDim.x)
    u1[c] = (float)acc[c] / denbas;
}

__global__ void k_finish_f64(const double* __restrict__ acc, int64_t g, float denbas,
                             float* __restrict__ u1) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g;
       c += (int64_t)gridDim.x * blockDim.x)
    u1[c] = (float)acc[c] / denbas;
}

// ------------------------------------------------------------ spatial bins
// Coarse binning of the store (bins of `bw` base cells) so a patch finds the
// particles near it without scanning all N (the reference tests every
// particle against every patch, grids.f:879-893).
struct Bins {
  int nb;          // bins per axis
  float xl, bsz;   // origin and bin size
  float eps;       // in bins: a particle this little below a bin's lower face is in it
  int32_t* start;  // nb^3+1
  int32_t* idx;    // particle indices grouped by bin
};

// A range's lower bound and the reference's own INT((v - patch corner) / cell)
// round differently, so a particle may belong to a unit though its coordinate
// lies a few spacings below the bound: with the faces on a common grid that is a
// few spacings below a bin.  Particles are therefore binned eps = nb 2^-20 up
// (the roundings add to less than 10 nb 2^-24), and a range runs from the bin of
// its lower bound to the bin of its upper bound moved up likewise.
__device__ __forceinline__ int bin_clamp(float t, int nb) {
  const int b = (int)floorf(t);
  return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}
__device__ __forceinline__ int bin_lo(const Bins& B, float v) { return bin_clamp((v - B.xl) / B.bsz, B.nb); }
__device__ __forceinline__ int bin_hi(const Bins& B, float v) { return bin_clamp((v - B.xl) / B.bsz + B.eps, B.nb); }

// Sort key of a particle: its bin, then `sub` bits per axis of its place
// inside the bin, interleaved (0: input order within a bin).  With sub bits
// the particles of one cell follow each other, so a warp that reads 32 of them
// meets few cells.
__device__ __forceinline__ uint32_t bin_key(const Bins& B, float x, float y, float z, int sub) {
  const float v[3] = {x, y, z};
  uint32_t b[3], low = 0;
  for (int a = 0; a < 3; a++) {
    const float t = (v[a] - B.xl) / B.bsz + B.eps;
    b[a] = (uint32_t)bin_clamp(t, B.nb);
    if (sub) {
      const int m = 1 << sub, q = (int)((t - (float)b[a]) * (float)m);
      const uint32_t u = (uint32_t)(q < 0 ? 0 : (q >= m ? m - 1 : q));
      for (int s = 0; s < sub; s++) low |= ((u >> s) & 1u) << (3 * s + a);
    }
  }
  return (((b[2] * (uint32_t)B.nb + b[1]) * (uint32_t)B.nb + b[0]) << (3 * sub)) | low;
}

__global__ void k_bin_keys(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                           int64_t n, Bins B, int sub, uint32_t* __restrict__ keys, int32_t* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = bin_key(B, x[i], y[i], z[i], sub);
    vals[i] = (int32_t)i;
  }
}

// First sorted position of every bin that holds particles; the others keep
// their initial n and take the next bin's start in the scan that follows.
__global__ void k_bin_heads(const uint32_t* __restrict__ keys, int64_t n, int sub, int32_t* __restrict__ start) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = keys[i] >> (3 * sub);
    if (i == 0 || (keys[i - 1] >> (3 * sub)) != b) start[b] = (int32_t)i;
  }
}

__global__ void k_fill_i32(int32_t* __restrict__ a, int64_t n, int32_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    a[i] = v;
}

struct MinI32 {
  __host__ __device__ int32_t operator()(int32_t a, int32_t b) const { return a < b ? a : b; }
};

// Where a density buffer lives: the call's arena, or density pool 0 when
// the patch deposit is deferred (buffers the deferred kernels read).
struct DAlloc {
  asohf_ctx* c;
  bool pool;
  void* get(size_t bytes) const { return pool ? dpool_alloc(c, 0, bytes) : arena_alloc(c, bytes); }
};

// start[b] = first position of bin b (from the sorted keys: the heads, then a
// minimum scan from the back; with an atomic count of every particle the bins
// of 56.6M particles took 2.33 ms, so 1.90), idx = the particles grouped by bin (a stable
// radix sort of (key, index): the same grouping on every run).
static int bin_key_bits(int64_t nbin) {
  int bits = 1;
  while ((1ll << bits) < nbin) bits++;
  return bits;
}

// Sub-cell bits per axis (at most `want`) that keep the key in 32 bits.
static int bin_sub(int64_t nbin, int want) {
  const int room = (32 - bin_key_bits(nbin)) / 3;
  return room < 0 ? 0 : (want < room ? want : room);
}

typedef thrust::reverse_iterator<int32_t*> RevI32;

static void bins_temp(int64_t n, int64_t nbin, int sub, size_t* scan_b, size_t* sort_b) {
  *scan_b = 0;
  *sort_b = 0;
  cub::DeviceScan::InclusiveScan(nullptr, *scan_b, RevI32(nullptr), RevI32(nullptr), MinI32(), (int)(nbin + 1));
  cub::DeviceRadixSort::SortPairs(nullptr, *sort_b, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                  (int32_t*)nullptr, (int)(n > 0 ? n : 1), 0, bin_key_bits(nbin) + 3 * sub);
}

static int64_t bins_per_axis(float lado0, float dx, int bw) {
  const int nx = (int)lrintf(lado0 / dx);
  const int nb = (nx + bw - 1) / bw;
  return nb < 1 ? 1 : nb;
}

static int build_bins(asohf_ctx* c, float lado0, float dx, int bw, Bins* B, DAlloc A = DAlloc{nullptr, false},
                      int want_sub = 0) {
  int64_t n = c->p.n;
  const int nb = (int)bins_per_axis(lado0, dx, bw);
  int64_t nbin = (int64_t)nb * nb * nb;
  const int sub = bin_sub(nbin, want_sub);
  B->nb = nb;
  B->xl = -lado0 / 2.0f;
  B->bsz = lado0 / (float)nb;
  B->eps = ldexpf((float)nb, -20);
  uint32_t* k0 = (uint32_t*)arena_alloc(c, 4 * n + 4);
  uint32_t* k1 = (uint32_t*)arena_alloc(c, 4 * n + 4);
  int32_t* v0 = (int32_t*)arena_alloc(c, 4 * n + 4);
  B->start = (int32_t*)(A.pool ? A.get(4 * (nbin + 1)) : arena_alloc(c, 4 * (nbin + 1)));
  B->idx = (int32_t*)arena_alloc(c, 4 * n + 4);
  size_t ts, tr;
  bins_temp(n, nbin, sub, &ts, &tr);
  void* t = arena_alloc(c, ts > tr ? ts : tr);
  if (!k0 || !k1 || !v0 || !B->start || !B->idx || !t) return ASOHF_ERR_CAPACITY;
  int kt_ = ktime_begin(c, "particle_bins");
  k_fill_i32<<<grid_for(nbin + 1, 256), 256, 0, c->stream>>>(B->start, nbin + 1, (int32_t)n);
  c->launches++;
  if (n > 0) {
    k_bin_keys<<<grid_for(n, 256), 256, 0, c->stream>>>(c->p.x, c->p.y, c->p.z, n, *B, sub, k0, v0);
    ASOHF_CUDA(cub::DeviceRadixSort::SortPairs(t, tr, k0, k1, v0, B->idx, (int)n, 0,
                                               bin_key_bits(nbin) + 3 * sub, c->stream));
    k_bin_heads<<<grid_for(n, 256), 256, 0, c->stream>>>(k1, n, sub, B->start);
    ASOHF_CUDA(cub::DeviceScan::InclusiveScan(t, ts, RevI32(B->start + nbin + 1), RevI32(B->start + nbin + 1),
                                              MinI32(), (int)(nbin + 1), c->stream));
    c->launches += 2;
  }
  ktime_end(c, kt_);
  return ASOHF_OK;
}

static size_t bins_bytes(int64_t n, float lado0, float dx, int bw, int want_sub = 0) {
  const int64_t nb = bins_per_axis(lado0, dx, bw), nbin = nb * nb * nb;
  size_t ts, tr;
  bins_temp(n, nbin, bin_sub(nbin, want_sub), &ts, &tr);
  return 16 * (size_t)n + 4 * (size_t)(nbin + 1) + (ts > tr ? ts : tr) + 8192;
}

// Device copy of the patch table.
struct DevMesh {
  int np;
  int32_t *nx, *ny, *nz, *level;
  float *rx, *ry, *rz;
};

static int upload_mesh(asohf_ctx* c, const asohf_mesh* mh, DevMesh* d, DAlloc A = DAlloc{nullptr, false}) {
  int np = 0;
  for (int ir = 1; ir <= mh->nl; ir++) np += mh->npatch[ir];
  d->np = np;
  if (np == 0) return ASOHF_OK;
  int base = mh->npatch[0];
  for (int q = 0; q < np; q++) {
    int ip = base + q;
    if (mh->patchnx[ip] < 1 || mh->patchnx[ip] > ASOHF_NAMRX || mh->patchny[ip] < 1 || mh->patchny[ip] > ASOHF_NAMRX ||
        mh->patchnz[ip] < 1 || mh->patchnz[ip] > ASOHF_NAMRX)
      return ASOHF_ERR_INVALID;
  }
  std::vector<int32_t> hi_v(4 * (size_t)np);
  std::vector<float> hf_v(3 * (size_t)np);
  int32_t* hi = hi_v.data();
  float* hf = hf_v.data();
  int q = 0;
  for (int ir = 1; ir <= mh->nl; ir++)
    for (int p = 0; p < mh->npatch[ir]; p++, q++) {
      int ip = base + q;
      hi[q] = mh->patchnx[ip];
      hi[np + q] = mh->patchny[ip];
      hi[2 * np + q] = mh->patchnz[ip];
      hi[3 * np + q] = ir;
      hf[q] = mh->patchrx[ip];
      hf[np + q] = mh->patchry[ip];
      hf[2 * np + q] = mh->patchrz[ip];
    }
  int32_t* di = (int32_t*)(A.pool ? A.get(16 * (size_t)np) : arena_alloc(c, 16 * (size_t)np));
  float* df = (float*)(A.pool ? A.get(12 * (size_t)np) : arena_alloc(c, 12 * (size_t)np));
  if (!di || !df) return ASOHF_ERR_CAPACITY;
  cudaMemcpyAsync(di, hi, 16 * (size_t)np, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(df, hf, 12 * (size_t)np, cudaMemcpyHostToDevice, c->stream);
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  d->nx = di; d->ny = di + np; d->nz = di + 2 * np; d->level = di + 3 * np;
  d->rx = df; d->ry = df + np; d->rz = df + 2 * np;
  return ASOHF_OK;
}

// ------------------------------------------------------------ staging
// The store in bin order as float4 (x, y, z, m) plus the species index (in the
// mass's place when all masses are equal), so a patch reads its candidates as
// contiguous runs (one run per (y, z) row of bins).
#define NA ASOHF_NAMRX

__global__ void k_bin_stage(const int32_t* __restrict__ idx, int64_t n, int64_t ndep, const float* __restrict__ x,
                            const float* __restrict__ y, const float* __restrict__ z, const float* __restrict__ m,
                            const float4* __restrict__ rows, const int64_t* __restrict__ esp_end,
                            float4* __restrict__ P, uint8_t* __restrict__ S, int spec_in_w) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    int p = idx[t];
    float4 v = rows ? rows[2 * (int64_t)p] : make_float4(x[p], y[p], z[p], m[p]);
    if (esp_end) {
      int s = 0;
      while (s < ASOHF_N_ESP - 1 && (int64_t)p >= esp_end[s]) s++;
      if ((int64_t)p >= ndep) s = 255;  // not deposited
      if (spec_in_w) v.w = __int_as_float(s);
      else S[t] = (uint8_t)s;
    }
    P[t] = v;
  }
}

// ------------------------------------------------------------ base deposit, equal masses
// With one particle mass every particle of a host cell deposits the same
// 27 REAL*4 terms, so the grid is the 27-point stencil of the host-cell
// counts: U1(c) = sum_o count(c - o) * t_o, each product exact in float64.
// P (the binned copy, species in w) where there is one: its order keeps the
// atomics of a warp on a few lines of the grid, where the store's is random.
// With the stencil below, 56.6M particles on 384^3 take 1.27 ms, 2.47 ms with
// counts in store order, 27 loads a cell and a float64 grid read back.
__global__ void k_base_counts(const float* __restrict__ x, const float* __restrict__ y,
                              const float* __restrict__ z, const float4* __restrict__ P, int64_t n, int nx,
                              float xl, float dx, int32_t* __restrict__ cnt, int* __restrict__ outside) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float px, py, pz;
    if (P) {
      const float4 p = P[i];
      if (__float_as_int(p.w) == 255) continue;  // not deposited
      px = p.x; py = p.y; pz = p.z;
    } else {
      px = x[i]; py = y[i]; pz = z[i];
    }
    int ix = (int)((px - xl) / dx) + 1;
    int jy = (int)((py - xl) / dx) + 1;
    int kz = (int)((pz - xl) / dx) + 1;
    if (ix >= 1 && ix <= nx && jy >= 1 && jy <= nx && kz >= 1 && kz <= nx)
      atomicAdd(&cnt[((int64_t)(kz - 1) * nx + (jy - 1)) * nx + (ix - 1)], 1);
    else
      *outside = 1;
  }
}

struct Terms8 {
  double t[8];  // t[dk*4 + dj*2 + di] = ((m*W(di))*W(dj))*W(dk) in REAL*4, offsets 0 and 1
};

// The kernel is symmetric (W(-1) = W(1)): the 27 terms take 8 values, so a
// cell needs the count sums of 8 neighbour patterns (integers) and 8 products.
// A thread marches along z over BS_Z planes, keeping the in-plane pattern sums
// of three, and writes U1 at once unless particles outside the box are still to
// be added: 9 loads a cell instead of 27, no index divisions, no float64 grid.
#define BS_X 32
#define BS_Y 8
#define BS_Z 16
__global__ void __launch_bounds__(BS_X* BS_Y)
k_base_stencil(const int32_t* __restrict__ cnt, int nx, Terms8 T, float denbas, const int* __restrict__ outside,
               double* __restrict__ acc, float* __restrict__ u1) {
  const int i = blockIdx.x * BS_X + threadIdx.x, j = blockIdx.y * BS_Y + threadIdx.y;  // 0-based
  if (i >= nx || j >= nx) return;
  const bool keep = *outside != 0;
  const int im = i == 0 ? nx - 1 : i - 1, ip = i == nx - 1 ? 0 : i + 1;
  const int64_t r0 = (int64_t)j * nx, rm = (int64_t)(j == 0 ? nx - 1 : j - 1) * nx,
                rp = (int64_t)(j == nx - 1 ? 0 : j + 1) * nx;
  auto plane = [&](int k, int* q) {  // centre, x pair, y pair, corners
    const int32_t* pl = cnt + (int64_t)(k < 0 ? nx - 1 : (k >= nx ? k - nx : k)) * nx * nx;
    q[0] = pl[r0 + i];
    q[1] = pl[r0 + im] + pl[r0 + ip];
    q[2] = pl[rm + i] + pl[rp + i];
    q[3] = (pl[rm + im] + pl[rm + ip]) + (pl[rp + im] + pl[rp + ip]);
  };
  const int k0 = blockIdx.z * BS_Z, k1 = min(k0 + BS_Z, nx);
  int a[4], b[4], c[4];
  plane(k0 - 1, a);
  plane(k0, b);
  for (int k = k0; k < k1; k++) {
    plane(k + 1, c);
    double s = 0.0;
    int any = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) any |= a[q] | b[q] | c[q];
    if (any) {
      const int c4 = a[0] + c[0], c5 = a[1] + c[1], c6 = a[2] + c[2], c7 = a[3] + c[3];
      s = (double)b[0] * T.t[0] + (double)b[1] * T.t[1] + (double)b[2] * T.t[2] + (double)b[3] * T.t[3] +
          (double)c4 * T.t[4] + (double)c5 * T.t[5] + (double)c6 * T.t[6] + (double)c7 * T.t[7];
    }
    const int64_t at = (int64_t)k * nx * nx + r0 + i;
    if (keep) acc[at] = s;
    else u1[at] = (float)s / denbas;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      a[q] = b[q];
      b[q] = c[q];
    }
  }
}

// ------------------------------------------------------------ patch deposit
// Work unit: PZ z-planes of one patch.  A unit's candidates are the particles
// of the bins that overlap the patch box extended by MAXKERNELEXT = DX
// (grids.f:837-893), restricted in z to the unit's planes +- DX; they are split
// into slices so that a dense unit is shared by several CTAs, whose sums meet in
// a float64 scratch slab.
#define PZ 4              // z planes per unit
#define PZ_BLOCK 256
#define NSLAB (NA / PZ)
// Slices are cut by work: the candidates, weighted by the width of their clouds
// in a sample of the unit's.  A slice holds the share that gives `items` of them
// an SM, between lo and hi, or a twelfth of an SM's work where that is more.
// Large slices cost least where every CTA has many units to take (the equal-mass
// kernel at 384^3 with 8192, 16384, 24576 and 32768: 17.5, 16.3, 15.9, 15.7 ms),
// small ones spread few units, or few with many wide clouds: DENSITY of 262144
// particles on 299 patches to level 3 takes 0.38 ms with their species (0.44 with
// slices of 24576) and 1.8 with one species (8.1); 2.1M on 2207 patches 1.45
// (1.42) and 7.4 (10.7).  Weights of 1, 8, 100 and 100 cut ordinary units too often
// (2.1M to level 6 1.82 ms, 1.80 so).  The units still go in order of their counts:
// in order of their work 56.6M particles took 25.7 ms, 25.3 so.
struct SliceRule {
  int items, lo, hi;  // hi also bounds the candidates: the equal-mass kernel counts a slice's in 16 bits
  int w[4];           // weight of a cloud of level 1 or less, 2, 3, 4 or more
};
static const SliceRule kSliceEq{3, 8192, 24576, {1, 4, 6, 6}}, kSliceAny{6, 2048, 24576, {1, 2, 4, 13}},
    kSliceUnits{6, 2048, 24576, {1, 1, 1, 1}};
#define SLICE_MIN 256  // candidates
#define UNITS_FEW 512
#define PROWS 128         // bin rows staged in shared memory at a time
#define AROW (NA + 5)     // accumulator row stride (doubles): rows shifted by 5 banks pairs
#define APLANE (NA * AROW)
#define ACC_N (PZ * APLANE)

// Offset of the centre of level l in the compact kernel table that stores
// levels 0, 1, ... back to back (2*2^l+1 entries each).
__host__ __device__ __forceinline__ int ktab_center(int l) { return 3 * (1 << l) - 2 + l; }
__host__ __device__ __forceinline__ int ktab_size(int lmax) { return (1 << (lmax + 2)) - 1 + lmax; }

struct UnitGeo {
  int ip, slab, n1, n2, n3, ir, zlo, zhi;
  float dxpa, xlfix, ylfix, zlfix, pxl, pyl, pzl, pxr, pyr, pzr;
  int bx0, bx1, by0, by1, bz0, bz1, nby, rows;
};

__device__ __forceinline__ void unit_geo(const DevMesh& M, const Bins& B, const int32_t* order, int u, float dx,
                                         UnitGeo& g) {
  g.ip = order[u / NSLAB];
  g.slab = u % NSLAB;
  g.n1 = M.nx[g.ip]; g.n2 = M.ny[g.ip]; g.n3 = M.nz[g.ip]; g.ir = M.level[g.ip];
  g.zlo = g.slab * PZ + 1;
  g.zhi = min(g.slab * PZ + PZ, g.n3);
  g.dxpa = dx / exp2f((float)g.ir);
  g.xlfix = M.rx[g.ip] - g.dxpa; g.ylfix = M.ry[g.ip] - g.dxpa; g.zlfix = M.rz[g.ip] - g.dxpa;
  g.pxl = g.xlfix - dx; g.pyl = g.ylfix - dx; g.pzl = g.zlfix - dx;
  g.pxr = (g.xlfix + (float)g.n1 * g.dxpa) + dx;
  g.pyr = (g.ylfix + (float)g.n2 * g.dxpa) + dx;
  g.pzr = (g.zlfix + (float)g.n3 * g.dxpa) + dx;
  g.bx0 = bin_lo(B, g.pxl); g.bx1 = bin_hi(B, g.pxr);
  g.by0 = bin_lo(B, g.pyl); g.by1 = bin_hi(B, g.pyr);
  // a cloud reaches at most 2^ir cells = DX from its host cell: planes
  // zlo..zhi take hosts with z in [zlfix + (zlo-1) dxpa - DX, zlfix + zhi dxpa + DX]
  float za = fmaxf(g.pzl, (g.zlfix + (float)(g.zlo - 1) * g.dxpa) - dx);
  float zb = fminf(g.pzr, (g.zlfix + (float)g.zhi * g.dxpa) + dx);
  g.bz0 = bin_lo(B, za); g.bz1 = bin_hi(B, zb);
  g.nby = g.by1 - g.by0 + 1;
  g.rows = (g.zlo > g.zhi) ? 0 : g.nby * (g.bz1 - g.bz0 + 1);
}

__device__ __forceinline__ void row_range(const Bins& B, const UnitGeo& g, int row, int* lo, int* len) {
  int bz = g.bz0 + row / g.nby, by = g.by0 + row % g.nby;
  int64_t rb = ((int64_t)bz * B.nb + by) * B.nb;
  int a = B.start[rb + g.bx0], b = B.start[rb + g.bx1 + 1];
  *lo = a;
  *len = b - a;
}

// Candidates of a unit (one warp per unit), as a sort key that puts the largest
// count first, and its work: candidates times their weights in a sample of two a
// row, in sixteenths.
template <typename F>
__device__ __forceinline__ void unit_count(const Bins& B, const UnitGeo& g, int u, int lane, F weight, uint32_t* work,
                                           uint32_t* key, int32_t* unit, int32_t* nm) {
  long long s = 0, w = 0;
  for (int r = lane; r < g.rows; r += 32) {
    int lo, len;
    row_range(B, g, r, &lo, &len);
    s += len;
    if (len > 0) w += ((long long)len * (weight(lo + len / 4) + weight(lo + (int)(3ll * len / 4))) + 1) / 2;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    w += __shfl_down_sync(0xffffffffu, w, o);
  }
  if (lane == 0) {
    w = (w + 15) / 16;
    key[u] = ~(uint32_t)(s < 0xffffffffll ? s : 0xffffffffll);
    work[u] = (uint32_t)(w < 0xffffffffll ? w : 0xffffffffll);
    unit[u] = u;
    if (u == 0) *nm = 0;
  }
}

// P holds the species in w, or S does (P null).
__global__ void k_patch_unit_counts(DevMesh M, Bins B, const int32_t* __restrict__ order, int nunits, float dx,
                                    const float4* __restrict__ P, const uint8_t* __restrict__ S, SliceRule R,
                                    uint32_t* __restrict__ work, uint32_t* __restrict__ key,
                                    int32_t* __restrict__ unit, int32_t* __restrict__ nm) {
  int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (u >= nunits) return;
  UnitGeo g;
  unit_geo(M, B, order, u, dx, g);
  auto weight = [&](int e) {
    const int s = P ? __float_as_int(P[e].w) : (int)S[e], l = s == 255 ? 0 : g.ir - s;
    return l <= 1 ? R.w[0] : (l == 2 ? R.w[1] : (l == 3 ? R.w[2] : R.w[3]));
  };
  unit_count(B, g, u, lane, weight, work, key, unit, nm);
}

struct PatchWork {
  const int2* items;         // (unit, slice)
  const int2* unit;          // per unit: scratch slab index (-1: one slice), candidates of a slice
  double* scratch;           // the unit's cells in float64, per multi-slice unit
  const int* nitems;         // of a grid that may be larger, or null
  __device__ bool past() const { return nitems && (int)blockIdx.x >= *nitems; }
};

// Rows r0 .. r0+nr-1 of a unit's bins: first entries and the running total of
// their lengths (whole CTA; the caller synchronises before and after).
__device__ __forceinline__ void stage_rows(const Bins& B, const UnitGeo& g, int r0, int nr, int* s_lo, int* s_pre) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int run = 0;
    for (int r = lane; r - lane < nr; r += 32) {
      int lo = 0, len = 0;
      if (r < nr) row_range(B, g, r0 + r, &lo, &len);
      int sc = len;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, sc, o);
        if (lane >= o) sc += y;
      }
      if (r < nr) {
        s_lo[r] = lo;
        s_pre[r + 1] = run + sc;
      }
      run += __shfl_sync(0xffffffffu, sc, 31);
    }
    if (lane == 0) s_pre[0] = 0;
  }
}

// Row of candidate v: the last row whose total before it is not above v.
__device__ __forceinline__ int find_row(const int* s_pre, int nr, int v) {
  int lo = 0, hi = nr - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_pre[mid] <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Work items of a patch deposit, built on the device: the units in order of
// falling candidate count, each cut into slices.  The host reads two numbers
// (items, units with several slices) to size the buffers.  (Counts to the host,
// sorted there and the lists sent back took 1.6 ms of the 37 ms of 12012 patches
// at 384^3; this takes under 0.1 ms.)  Of up to UNITS_FEW units one CTA makes the
// list in unit order, in buffers of the largest size it can take, and the host
// reads nothing: the mesh counts of 7 patches over 32768 particles 0.21 ms, 0.25
// with the sort, the scan and the wait.
struct UnitList {
  int nunits = 0, nitems = 0, nmulti = 0;    // (bounds of the two where few)
  bool few = false;
  SliceRule rule{};
  uint32_t* work = nullptr;                  // by unit
  uint32_t *key = nullptr, *key2 = nullptr;  // ~count, by unit and sorted
  int32_t *unit = nullptr, *ord = nullptr;
  int32_t *ns = nullptr, *off = nullptr;     // slices of each sorted unit, and the sum before it
  int32_t *slab = nullptr, *nm = nullptr;    // scratch slab of each, and the slabs in all
  void* tmp = nullptr;
  size_t sort_b = 0, scan_b = 0;
};

static void unit_list_temp(int nunits, size_t* sort_b, size_t* scan_b) {
  *sort_b = *scan_b = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, *sort_b, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                  (int32_t*)nullptr, nunits > 0 ? nunits : 1);
  cub::DeviceScan::ExclusiveSum(nullptr, *scan_b, (int32_t*)nullptr, (int32_t*)nullptr, nunits + 1);
}

static size_t unit_list_bytes(int nunits) {
  size_t a, b;
  unit_list_temp(nunits, &a, &b);
  return 40 * (size_t)nunits + (a > b ? a : b) + 16 * 256;
}

static int unit_list_begin(asohf_ctx* c, int nunits, UnitList* U) {
  U->nunits = nunits;
  const size_t b = 4 * (size_t)nunits + 4;
  U->work = (uint32_t*)arena_alloc(c, b);
  U->key = (uint32_t*)arena_alloc(c, b);
  U->key2 = (uint32_t*)arena_alloc(c, b);
  U->unit = (int32_t*)arena_alloc(c, b);
  U->ord = (int32_t*)arena_alloc(c, b);
  U->ns = (int32_t*)arena_alloc(c, b);
  U->off = (int32_t*)arena_alloc(c, b);
  U->slab = (int32_t*)arena_alloc(c, b);
  U->nm = (int32_t*)arena_alloc(c, 4);
  unit_list_temp(nunits, &U->sort_b, &U->scan_b);
  U->tmp = arena_alloc(c, U->sort_b > U->scan_b ? U->sort_b : U->scan_b);
  return U->work && U->key && U->key2 && U->unit && U->ord && U->ns && U->off && U->slab && U->nm && U->tmp
             ? ASOHF_OK
             : ASOHF_ERR_CAPACITY;
}

// The share of work a slice holds, from that of all units (sixteenths).
__device__ __forceinline__ double slice_share(double sum, int sms, const SliceRule& R) {
  const double sm = 16.0 * sum / sms;  // an SM's work
  return fmax(fmin(fmax(sm / R.items, (double)R.lo), (double)R.hi), sm / 12.0);
}

// Slices of a unit: at most 1 + work/share + cnt/hi.
__device__ __forceinline__ int unit_slices(uint32_t cnt, uint32_t work, double share, const SliceRule& R) {
  const double most = fmax(1.0, (double)(cnt / SLICE_MIN));
  const int k = (int)fmin(most, ceil(16.0 * (double)work / share));
  return max(max(k, 1), (int)((cnt + (uint64_t)R.hi - 1) / R.hi));
}

// Slices of the sorted units (256 threads).  Every CTA sums the work over up to
// 1024 units, else over 1024 or more evenly spaced in the sorted order (the counts
// fall steadily) times their distance.
__global__ void k_unit_slices(const uint32_t* __restrict__ key, const int32_t* __restrict__ ord,
                              const uint32_t* __restrict__ work, int n, int sms, SliceRule R, int32_t* __restrict__ ns,
                              int32_t* __restrict__ slab, int32_t* __restrict__ nm) {
  __shared__ double s_sum[32];
  const int step = n > 1024 ? n / 1024 : 1;
  double sum = 0.0;
  for (int64_t q = (int64_t)threadIdx.x * step; q < n; q += 256 * (int64_t)step) sum += (double)work[ord[q]];
  const double share = slice_share(block_sum_d(sum, s_sum) * step, sms, R);
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > n) return;
  const int k = r < n ? unit_slices(~key[r], work[ord[r]], share, R) : 0;
  ns[r] = k;
  if (r < n) slab[r] = k > 1 ? atomicAdd(nm, 1) : -1;
}

// After the counts: the sort, the slices and their sum; reads the totals.
static int unit_list_size(asohf_ctx* c, UnitList* U, SliceRule R) {
  const int n = U->nunits;
  const int64_t whole = c->p.n * n / R.hi;  // slices of R.hi candidates, at most
  U->few = n <= UNITS_FEW && whole < 4096;
  U->rule = R;
  if (U->few) {
    U->nitems = n + 12 * c->num_sms + (int)whole + 16;
    U->nmulti = n;
    return ASOHF_OK;
  }
  ASOHF_CUDA(cub::DeviceRadixSort::SortPairs(U->tmp, U->sort_b, U->key, U->key2, U->unit, U->ord, n, 0, 32,
                                             c->stream));
  k_unit_slices<<<n / 256 + 1, 256, 0, c->stream>>>(U->key2, U->ord, U->work, n, c->num_sms, R, U->ns, U->slab,
                                                     U->nm);
  ASOHF_CUDA(cub::DeviceScan::ExclusiveSum(U->tmp, U->scan_b, U->ns, U->off, n + 1, c->stream));
  c->launches++;
  int32_t h[2];
  ASOHF_CUDA(cudaMemcpyAsync(&h[0], U->off + n, 4, cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaMemcpyAsync(&h[1], U->nm, 4, cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  U->nitems = h[0];
  U->nmulti = h[1];
  return ASOHF_OK;
}

static size_t unit_work_bytes(const UnitList& U, int unit_cells) {
  return sizeof(int2) * (size_t)U.nitems + 4 * (size_t)U.nmulti + 8 * (size_t)unit_cells * U.nmulti + 4 * 256;
}

// multi: the unit of each scratch slab (-1: the slab is not used).
__global__ void k_unit_items(const int32_t* __restrict__ ord, const int32_t* __restrict__ ns,
                             const int32_t* __restrict__ off, const int32_t* __restrict__ slab,
                             const uint32_t* __restrict__ key, int n, int2* __restrict__ items,
                             int2* __restrict__ unit, int32_t* __restrict__ multi) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int u = ord[r], k = ns[r], o = off[r], l = slab[r];
  for (int q = 0; q < k; q++) items[o + q] = make_int2(u, q);
  unit[u] = make_int2(l, (int)((~key[r] + (uint64_t)k - 1) / k));
  if (l >= 0) multi[l] = u;
}

// The list of few units, in unit order (one CTA of UNITS_FEW threads).
__global__ void __launch_bounds__(UNITS_FEW)
k_unit_list_few(const uint32_t* __restrict__ key, const uint32_t* __restrict__ work, int n, int sms, SliceRule R, int cap,
                int2* __restrict__ items, int2* __restrict__ unit, int32_t* __restrict__ multi,
                int* __restrict__ nitems) {
  __shared__ double s_sum[32];
  __shared__ int s_run[32];
  const int u = threadIdx.x, lane = u & 31;
  const double share = slice_share(block_sum_d(u < n ? (double)work[u] : 0.0, s_sum), sms, R);
  const int k = u < n ? unit_slices(~key[u], work[u], share, R) : 0;
  int end = k;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += v;
  }
  if (lane == 31) s_run[u >> 5] = end;
  __syncthreads();
  for (int w = 0; w < u >> 5; w++) end += s_run[w];
  if (u == UNITS_FEW - 1) *nitems = min(end, cap);
  if (u >= n) return;
  for (int q = 0; q < k && end - k + q < cap; q++) items[end - k + q] = make_int2(u, q);
  unit[u] = make_int2(k > 1 ? u : -1, (int)((~key[u] + (uint64_t)k - 1) / k));
  multi[u] = k > 1 ? u : -1;
}

// The items, scratch slabs (cleared) and slab indices, in buffers of the
// caller's: `walloc` for what unit_work_bytes counts, `salloc` for 8 bytes a unit and 8.
template <typename FW, typename FS>
static int unit_list_fill(asohf_ctx* c, const UnitList& U, int unit_cells, FW walloc, FS salloc, PatchWork* W,
                          int32_t** multi) {
  int2* items = (int2*)walloc(sizeof(int2) * (size_t)U.nitems);
  *multi = (int32_t*)walloc(4 * (size_t)(U.nmulti > 0 ? U.nmulti : 1));
  const size_t sb = 8 * (size_t)unit_cells * U.nmulti;
  W->scratch = (double*)walloc(sb > 0 ? sb : 8);
  int2* unit = (int2*)salloc(8 * (size_t)U.nunits + 8);
  int* nitems = (int*)(unit + U.nunits);
  if (!items || !*multi || !W->scratch || !unit) return ASOHF_ERR_CAPACITY;
  if (sb) ASOHF_CUDA(cudaMemsetAsync(W->scratch, 0, sb, c->stream));
  W->nitems = U.few ? nitems : nullptr;
  if (U.few)
    k_unit_list_few<<<1, UNITS_FEW, 0, c->stream>>>(U.key, U.work, U.nunits, c->num_sms, U.rule, U.nitems, items, unit,
                                                    *multi, nitems);
  else
    k_unit_items<<<(U.nunits + 255) / 256, 256, 0, c->stream>>>(U.ord, U.ns, U.off, U.slab, U.key2, U.nunits, items,
                                                                unit, *multi);
  c->launches++;
  W->items = items;
  W->unit = unit;
  return ASOHF_OK;
}

// One work item (a slice of one PZ-plane unit of a patch), equal masses.  The
// unit's sums live in registers: lane i of warp w holds cells (i, 4w .. 4w+3,
// every plane) in float64, so clouds are added without atomics.  Hosts of level
// 0 and 1 (most hits) are counted, both levels in the halves of one word a cell
// (a slice holds at most kSliceEq.hi hosts, so no half and no sum of counts
// overflows), and spread by a stencil at the end: with a kernel symmetric in
// each axis the (2r+1)^3 terms of a level take (r+1)^3 values t(|di|, |dj|,
// |dk|), each formed once.  Wider clouds are listed by the scan and added by
// the warps whose rows they meet.
//
// Float64 conversions run at 16 lanes a clock and SM and shared-memory float64
// atomics (compare and swap) at 4.7, additions at 61.  A positive normal REAL*4
// term is widened by one integer product, its bits times 2^29, which is the
// term times 2^-896 exactly; the sums are scaled back at the end.
//
// Measured at 56.6M particles, 12012 patches (96096 units, 698M candidates, 166M
// hits): 15.9 ms; 21.7 ms with every hit above level 0 added by shared-memory
// atomics.  About 6 ms are the scan, 4.5 the level-2 clouds, 2.6 the stencil, 2
// the wider clouds, 1.5 clearing and writing; bound by instruction issue and
// the latency of short lists (24 warps an SM, registers and shared memory).
#define SCALE_UP 0x1p896
#define CG (NA + 4)               // count grid rows: x, y in [-1, NA+2]
#define CGP (PZ + 4)              // its planes, z in [zlo-2, zhi+2]
#define ROUND (PZ_BLOCK * 2)      // candidates scanned between two looks at the lists
#define LCAP (2 * ROUND)          // listed clouds, added when another round might not fit
// Level-2 clouds of one mass (9^3 cells, the most of the listed ones): their
// terms as a table t[|di|][|dj|][dk], 0 past the cloud, 4 copies shifted by a
// plane each so that the terms of a unit's 4 planes are one 16-byte read, and
// their list sorted by (eighth columns, quarter rows) of the host.  A cloud of
// columns 8b-7 .. 8b+8 leaves most of a warp's 32 columns idle, so a warp adds
// clouds of the host blocks 0, 2, 4 together, each on its own lanes, then those
// of blocks 1 and 3.
#define T2R 20                    // floats a row of the table: 16 used, banks spread
#define T2A (6 * T2R)
#define T2COPY (6 * T2A)
#define NB2 50                    // 5 column blocks of 8 hosts x 10 row blocks of 4

__device__ __forceinline__ double widen(float t) {
  unsigned long long w;
  asm("mul.wide.u32 %0, %1, 0x20000000;" : "=l"(w) : "r"(__float_as_uint(t)));
  return __longlong_as_double((long long)w);
}

// a count below 2^32 as float64: the low word of 2^52 + v
__device__ __forceinline__ double count_d(uint32_t v) {
  return __hiloint2double(0x43300000, (int)v) - 4503599627370496.0;
}

// floor(v / d) of the rounded quotient: the product with rd = 1/d, below 1000
// within 3e-4 of it, decides unless it lies within 1e-3 of an integer
__device__ __forceinline__ int floor_div(float v, float d, float rd) {
  const float r = v * rd;
  float f = floorf(r);
  if (fabsf(r - rintf(r)) < 1e-3f || fabsf(r) > 1000.0f) f = floorf(v / d);
  return (int)f;
}

__global__ void __launch_bounds__(PZ_BLOCK, 3)
k_density_patches_eq(DevMesh M, Bins B, const float4* __restrict__ P, const int32_t* __restrict__ order, PatchWork W,
                     float dx, const float* __restrict__ kernels,
                     float meq, const float* __restrict__ t2g, float* __restrict__ u11,
                     const float* __restrict__ denbas_lev) {
  extern __shared__ uint4 dyn[];
  uint32_t* cnt = (uint32_t*)dyn;             // counts[CGP][CG][CG]
  float* t2 = (float*)(cnt + CGP * CG * CG);  // the level-2 table
  float* ktab = t2 + 4 * T2COPY;              // the kernels
  __shared__ int s_lo[PROWS], s_pre[PROWS + 1], s_nlist, s_any[2];
  __shared__ unsigned long long s_list[LCAP];
  __shared__ double s_t0[8], s_t1[27];
  __shared__ unsigned short s_l2[LCAP], s_l2s[LCAP + 1];  // listed level-2 clouds, and sorted
  __shared__ int s_nl2, s_off2[NB2 + 1], s_cur2[NB2];
  const unsigned FULL = 0xffffffffu;
  if (W.past()) return;
  const int2 it = W.items[blockIdx.x];
  UnitGeo g;
  unit_geo(M, B, order, it.x, dx, g);
  float* out = u11 + (size_t)g.ip * NA * NA * NA + (size_t)g.slab * PZ * NA * NA;
  if (g.zlo > g.zhi) {  // planes past the patch
    for (int q = threadIdx.x; q < NA * NA * PZ; q += blockDim.x) out[q] = 0.0f;
    return;
  }
  for (int q = threadIdx.x; q < CGP * CG * CG; q += blockDim.x) cnt[q] = 0;
  for (int l = 0; l <= g.ir; l++) {
    int nk = 1 << l, c0 = ktab_center(l);
    for (int i = threadIdx.x - nk; i <= nk; i += blockDim.x)
      ktab[c0 + i] = kernels[(size_t)l * KW + ASOHF_NMAX_KERNELS + i];
  }
  if (threadIdx.x < 2) s_any[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_nlist = s_nl2 = 0;
  __syncthreads();
  if (threadIdx.x < 35) {  // the distinct terms of levels 0 and 1
    const int l = threadIdx.x < 27 ? 1 : 0, q = l ? threadIdx.x : threadIdx.x - 27, b = l ? 3 : 2;
    if (l <= g.ir) {
      const float* kc = ktab + ktab_center(l);
      (l ? s_t1 : s_t0)[q] =
          widen(__fmul_rn(__fmul_rn(__fmul_rn(meq, kc[q % b]), kc[(q / b) % b]), kc[q / (b * b)]));
    }
  }
  if (g.ir >= 2)
    for (int q = threadIdx.x; q < T2COPY; q += blockDim.x) ((float4*)t2)[q] = ((const float4*)t2g)[q];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j0 = 4 * warp + 1;  // the warp's rows j0 .. j0+3
  double acc[4][PZ];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int p = 0; p < PZ; p++) acc[q][p] = 0.0;
  const float rdx = 1.0f / g.dxpa;
  // the listed clouds on the warp's rows
  auto add_listed = [&](int nl) {
    for (int e0 = 0; e0 < nl; e0 += 32) {
      unsigned todo = 0;
      {
        bool mine = false;
        if (e0 + lane < nl) {
          const unsigned long long e = s_list[e0 + lane];
          const int jy = (int)((e >> 32) & 0xffff) - 1024, nk = 1 << (int)(e & 0xffff);
          mine = jy - nk <= j0 + 3 && jy + nk >= j0 && j0 <= g.n2;
        }
        todo = __ballot_sync(FULL, mine);
      }
      while (todo) {
        const int src = e0 + __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned long long e = s_list[src];
        const int ix = (int)(e >> 48) - 1024, jy = (int)((e >> 32) & 0xffff) - 1024;
        const int kz = (int)((e >> 16) & 0xffff) - 1024, lev = (int)(e & 0xffff), nk = 1 << lev;
        const float* kc = ktab + ktab_center(lev);
        const int ox = lane + 1 - ix;
        const float bx = ox >= -nk && ox <= nk ? __fmul_rn(meq, kc[ox]) : 0.0f;
        float wz[PZ];
#pragma unroll
        for (int p = 0; p < PZ; p++) {
          const int oz = g.zlo + p - kz;
          wz[p] = oz >= -nk && oz <= nk ? kc[oz] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int oy = j0 + q - jy;
          if (oy >= -nk && oy <= nk) {
            const float bw = __fmul_rn(bx, kc[oy]);
#pragma unroll
            for (int p = 0; p < PZ; p++) acc[q][p] += widen(__fmul_rn(bw, wz[p]));
          }
        }
      }
    }
  };
  // the level-2 list: counting sort by block, then every warp its three row
  // blocks (hosts within 4 rows of its own), several column blocks at a time
  auto add_level2 = [&](int n) {
    if (n == 0) return;
    for (int q = threadIdx.x; q < NB2; q += blockDim.x) s_cur2[q] = 0;
    __syncthreads();
    auto block = [](unsigned e) { return (int)((e >> 13) * 10 + ((e >> 6) & 15)); };
    for (int q = threadIdx.x; q < n; q += blockDim.x) atomicAdd(&s_cur2[block(s_l2[q])], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
      int run = 0;
      for (int q = lane; q - lane < NB2; q += 32) {
        const int v = q < NB2 ? s_cur2[q] : 0;
        int sc = v;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL, sc, o);
          if (lane >= o) sc += y;
        }
        if (q < NB2) s_off2[q] = s_cur2[q] = run + sc - v;
        run += __shfl_sync(FULL, sc, 31);
      }
      if (lane == 0) s_off2[NB2] = run;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const unsigned short e = s_l2[q];
      s_l2s[atomicAdd(&s_cur2[block(e)], 1)] = e;
    }
    __syncthreads();
#pragma unroll 1
    for (int phase = 0; phase < 2; phase++) {
      const int bin = phase == 0 ? (lane < 8 ? 0 : (lane < 24 ? 2 : 4)) : (lane < 16 ? 1 : 3);
      const int lo = s_off2[bin * 10 + warp], len = s_off2[bin * 10 + warp + 3] - lo;
      const int most = __reduce_max_sync(FULL, len);
      for (int q = 0; q < most; q++) {
        const unsigned e = s_l2s[q < len ? lo + q : lo];
        const int a = q < len ? min(abs(lane + 4 - (int)(e >> 10)), 5) : 5;
        const int dz = 11 - (int)(e & 15), dj = j0 + 3 - (int)((e >> 4) & 63);
        const float* t = t2 + (dz & 3) * T2COPY + a * T2A + (dz & ~3);
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const float4 v = *(const float4*)(t + min(abs(dj + r), 5) * T2R);
          acc[r][0] += widen(v.x);
          acc[r][1] += widen(v.y);
          acc[r][2] += widen(v.z);
          acc[r][3] += widen(v.w);
        }
      }
    }
  };
  const int slice = W.unit[it.x].y;
  const int64_t v0 = (int64_t)it.y * slice, v1 = v0 + slice;
  int64_t vbase = 0;
  for (int r0 = 0; r0 < g.rows; r0 += PROWS) {
    const int nr = min(PROWS, g.rows - r0);
    __syncthreads();
    stage_rows(B, g, r0, nr, s_lo, s_pre);
    __syncthreads();
    const int tot = s_pre[nr];
    const int b = (int)(min(v1, vbase + tot) - vbase);
    const int a = (int)(max(v0, vbase) - vbase);
    for (int rb = a; rb < b; rb += ROUND) {  // 64 candidates a warp
      const int cb = rb + warp * 64, ce = min(cb + 63, b - 1);
      if (cb <= ce) {
        // rows of the warp's first and last candidates
        int c0 = 0, c1 = 0;
        for (int r = 1 + lane; r <= nr; r += 32) {
          const int sp = s_pre[r];
          c0 += sp <= cb;
          c1 += sp <= ce;
        }
        int row0 = (int)__reduce_add_sync(FULL, (unsigned)c0);
        const int row1 = (int)__reduce_add_sync(FULL, (unsigned)c1);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int v = cb + 32 * h + lane;
          int ix = 0, jy = 0, kz = 0, lev = -1;
          if (v <= ce) {
            int row = row0, hi = row1;
            while (row < hi) {
              const int mid = (row + hi + 1) >> 1;
              if (s_pre[mid] <= v) row = mid; else hi = mid - 1;
            }
            row0 = row;
            const int e = s_lo[row] + (v - s_pre[row]);
            const float4 q = P[e];
            const int s = __float_as_int(q.w);
            if (s != 255 && g.pxl < q.x && q.x < g.pxr && g.pyl < q.y && q.y < g.pyr && g.pzl < q.z && q.z < g.pzr) {
              const int l = max(g.ir - s, 0), nk = 1 << l;
              ix = floor_div(q.x - g.xlfix, g.dxpa, rdx) + 1;
              jy = floor_div(q.y - g.ylfix, g.dxpa, rdx) + 1;
              kz = floor_div(q.z - g.zlfix, g.dxpa, rdx) + 1;
              if (!(ix - nk > g.n1 || ix + nk < 1 || jy - nk > g.n2 || jy + nk < 1) && kz - nk <= g.zhi &&
                  kz + nk >= g.zlo) {
                lev = l;
              }
            }
          }
          if (lev == 0 || lev == 1) {
            atomicAdd(&cnt[((kz - g.zlo + 2) * CG + (jy + 1)) * CG + (ix + 1)], lev ? 0x10000u : 1u);
            s_any[lev] = 1;
          }
          {
            const unsigned two = __ballot_sync(FULL, lev == 2);
            if (two) {
              int o = 0;
              if (lane == 0) o = atomicAdd(&s_nl2, __popc(two));
              o = __shfl_sync(FULL, o, 0) + __popc(two & ((1u << lane) - 1u));
              if (lev == 2)
                s_l2[o] = (unsigned short)(((ix + 3) << 10) | ((jy + 3) << 4) | (kz - g.zlo + 4));
            }
            if (lev == 2) lev = -1;
          }
          const unsigned wide = __ballot_sync(FULL, lev >= 2);
          if (wide) {
            int o = 0;
            if (lane == 0) o = atomicAdd(&s_nlist, __popc(wide));
            o = __shfl_sync(FULL, o, 0) + __popc(wide & ((1u << lane) - 1u));
            if (lev >= 2) {
              s_list[o] = (unsigned long long)(uint32_t)(((ix + 1024) << 16) | (jy + 1024)) << 32 |
                          (uint32_t)(((kz + 1024) << 16) | lev);
            }
          }
        }
      }
      __syncthreads();
      const int nl = s_nlist, nl2 = s_nl2;
      __syncthreads();
      if (nl > LCAP - ROUND || nl2 > LCAP - ROUND) {
        add_listed(nl);
        add_level2(nl2);
        __syncthreads();
        if (threadIdx.x == 0) s_nlist = s_nl2 = 0;
        __syncthreads();
      }
    }
    vbase += tot;
  }
  __syncthreads();
  add_listed(s_nlist);
  add_level2(s_nl2);
  if (s_any[0] | s_any[1]) {
    const bool any0 = s_any[0] != 0, any1 = s_any[1] != 0;
#pragma unroll 1
    for (int a = 0; a < 3; a++) {  // |di|
#pragma unroll
      for (int pl = 0; pl < CGP; pl++) {
        uint32_t X[8];  // rows j0-2 .. j0+5: the counts at -a and +a
#pragma unroll
        for (int r = 0; r < 8; r++) {
          const uint32_t* c = cnt + (pl * CG + (4 * warp + r)) * CG + lane + 2;
          X[r] = a == 0 ? c[0] : c[-a] + c[a];
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int bb = 0; bb < 3; bb++) {  // |dj|
            const uint32_t Y = bb == 0 ? X[q + 2] : X[q + 2 - bb] + X[q + 2 + bb];
            if (any1) {
              const double d1 = count_d(Y >> 16);
#pragma unroll
              for (int p = 0; p < PZ; p++) {
                const int gz = pl - 2 - p < 0 ? p + 2 - pl : pl - 2 - p;  // |dk|
                if (gz <= 2) acc[q][p] = __fma_rn(d1, s_t1[gz * 9 + bb * 3 + a], acc[q][p]);
              }
            }
            if (any0 && bb < 2 && a < 2 && pl >= 1 && pl <= CGP - 2) {
              const double d0 = count_d(Y & 0xffffu);
#pragma unroll
              for (int p = 0; p < PZ; p++) {
                const int gz = pl - 2 - p < 0 ? p + 2 - pl : pl - 2 - p;
                if (gz <= 1) acc[q][p] = __fma_rn(d0, s_t0[gz * 4 + bb * 2 + a], acc[q][p]);
              }
            }
          }
      }
    }
  }
  const int sidx = W.unit[it.x].x;
  const float den = denbas_lev[g.ir];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int p = 0; p < PZ; p++) {
      const int j = j0 - 1 + q, at = (p * NA + j) * NA + lane;  // 0-based cell (lane, j, slab*PZ + p)
      const double s = acc[q][p] * SCALE_UP;
      if (sidx < 0)
        out[at] = lane < g.n1 && j < g.n2 && g.slab * PZ + p < g.n3 ? (float)s / den : 0.0f;
      else if (s != 0.0)  // one slice of a shared unit
        atomicAdd(&W.scratch[(size_t)sidx * NA * NA * PZ + at], s);
    }
}

// One work item, any masses: float64 sums in shared memory, one cloud a warp
// step, hits with the same host cell, level and mass once with their number as
// factor; the binned order keeps a cell's particles together, so a warp's hits
// fall into few groups (0.80 ms for 1.4M particles of two masses on 888 patches,
// 1.24 with input order inside the bins).  (The registers and lists of the
// equal-mass kernel measured slower here, 1.64 against 1.24 ms: without counts
// and tables every hit is listed or added by itself.)
__global__ void __launch_bounds__(PZ_BLOCK, 3)
k_density_patches(DevMesh M, Bins B, const float4* __restrict__ P, const uint8_t* __restrict__ S,
                  const int32_t* __restrict__ order, PatchWork W, float dx, const float* __restrict__ kernels,
                  float* __restrict__ u11, const float* __restrict__ denbas_lev) {
  extern __shared__ double acc[];  // ACC_N doubles (padded rows), kernel table
  float* ktab = (float*)(acc + ACC_N);
  if (W.past()) return;
  const int2 it = W.items[blockIdx.x];
  __shared__ int s_lo[PROWS], s_pre[PROWS + 1], s_next;
  __shared__ float s_rcp[NA + 1];  // 1/n for the clipped cloud widths n <= NA
  UnitGeo g;
  unit_geo(M, B, order, it.x, dx, g);
  float* out = u11 + (size_t)g.ip * NA * NA * NA + (size_t)g.slab * PZ * NA * NA;
  if (g.zlo > g.zhi) {  // planes past the patch
    for (int q = threadIdx.x; q < NA * NA * PZ; q += blockDim.x) out[q] = 0.0f;
    return;
  }
  for (int q = threadIdx.x; q < ACC_N; q += blockDim.x) acc[q] = 0.0;
  for (int l = 0; l <= g.ir; l++) {
    int nk = 1 << l, c0 = ktab_center(l);
    for (int i = threadIdx.x - nk; i <= nk; i += blockDim.x)
      ktab[c0 + i] = kernels[(size_t)l * KW + ASOHF_NMAX_KERNELS + i];
  }
  if (threadIdx.x >= 1 && threadIdx.x <= NA) s_rcp[threadIdx.x] = 1.0f / (float)threadIdx.x;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int slice = W.unit[it.x].y;
  const int64_t v0 = (int64_t)it.y * slice, v1 = v0 + slice;
  int64_t vbase = 0;
  for (int r0 = 0; r0 < g.rows; r0 += PROWS) {
    int nr = min(PROWS, g.rows - r0);
    __syncthreads();
    stage_rows(B, g, r0, nr, s_lo, s_pre);
    if (threadIdx.x == 0) s_next = (int)(max(v0, vbase) - vbase);  // this slice's first candidate in these rows
    __syncthreads();
    const int tot = s_pre[nr];
    const int b = (int)(min(v1, vbase + tot) - vbase);
    // warps take 32 candidates at a time from a shared counter: a warp that
    // met wide clouds takes fewer
    for (;;) {
      int cbase = 0;
      if (lane == 0) cbase = atomicAdd(&s_next, 32);
      cbase = __shfl_sync(0xffffffffu, cbase, 0);
      if (cbase >= b) break;
      const int v = cbase + lane, vlast = min(cbase + 31, b - 1);
      // rows of the warp's first and last candidates (rows whose start is
      // not above them), then each lane's row between the two
      int c0 = 0, c1 = 0;
      for (int r = 1 + lane; r <= nr; r += 32) {
        int sp = s_pre[r];
        c0 += sp <= cbase;
        c1 += sp <= vlast;
      }
      int row = (int)__reduce_add_sync(0xffffffffu, (unsigned)c0);
      int rhi = (int)__reduce_add_sync(0xffffffffu, (unsigned)c1);
      while (row < rhi) {
        int mid = (row + rhi + 1) >> 1;
        if (s_pre[mid] <= v) row = mid; else rhi = mid - 1;
      }
      bool hit = false;
      float mp = 0.f;
      int ix = 0, jy = 0, kz = 0, lev = 0;
      if (v < b) {
        int e = s_lo[row] + (v - s_pre[row]);
        int s = S[e];
        float4 q = P[e];
        if (s != 255 && g.pxl < q.x && q.x < g.pxr && g.pyl < q.y && q.y < g.pyr && g.pzl < q.z && q.z < g.pzr) {
          lev = g.ir - s;
          if (lev < 0) lev = 0;
          int nk = 1 << lev;
          ix = (int)floorf((q.x - g.xlfix) / g.dxpa) + 1;
          jy = (int)floorf((q.y - g.ylfix) / g.dxpa) + 1;
          kz = (int)floorf((q.z - g.zlfix) / g.dxpa) + 1;
          if (!(ix - nk > g.n1 || ix + nk < 1 || jy - nk > g.n2 || jy + nk < 1 || kz - nk > g.n3 || kz + nk < 1) &&
              max(max(kz - nk, 1), g.zlo) <= min(min(kz + nk, g.n3), g.zhi)) {
            mp = q.w;
            hit = true;
          }
        }
      }
      unsigned long long key =
          hit ? ((unsigned long long)(ix + 1024) << 52) | ((unsigned long long)(jy + 1024) << 41) |
                    ((unsigned long long)(kz + 1024) << 30) | ((unsigned long long)lev << 26) |
                    (unsigned long long)(__float_as_uint(mp) >> 6)
              : ~0ull - (unsigned long long)lane;
      // hits of one host cell, level and mass deposit once with the group size as factor
      unsigned grp = 1u << lane;
      if (__popc(__ballot_sync(0xffffffffu, hit)) > 1) grp = __match_any_sync(0xffffffffu, key);
      if (hit && (grp & (grp - 1))) {  // the key keeps 26 bits of the mass: confirm equal masses
        float m0 = __shfl_sync(grp, mp, __ffs(grp) - 1);
        unsigned same = __ballot_sync(grp, mp == m0);
        if (same != grp) grp = 1u << lane;
      }
      // host cell (11 bits per axis, offset 1024), level and group size of each hit
      const int pxy = (ix + 1024) | ((jy + 1024) << 16);
      const int pzl = (kz + 1024) | (lev << 16) | (__popc(grp) << 24);
      unsigned hm = __ballot_sync(0xffffffffu, hit && lane == __ffs(grp) - 1);
      while (hm) {
        int src = __ffs(hm) - 1;
        hm &= hm - 1;
        const float wm = __shfl_sync(0xffffffffu, mp, src);
        const int wxy = __shfl_sync(0xffffffffu, pxy, src), wzl = __shfl_sync(0xffffffffu, pzl, src);
        const int wix = (wxy & 0xffff) - 1024, wjy = (wxy >> 16) - 1024, wkz = (wzl & 0xffff) - 1024;
        const int wlev = (wzl >> 16) & 0xff, nk = 1 << wlev;
        const double wc = (double)(wzl >> 24);
        // the cloud clipped to the patch and to the unit's planes
        const int wi1 = max(wix - nk, 1), wj1 = max(wjy - nk, 1), wk1 = max(max(wkz - nk, 1), g.zlo);
        const int wdi = min(wix + nk, g.n1) - wi1 + 1, wdj = min(wjy + nk, g.n2) - wj1 + 1;
        const int wdk = min(min(wkz + nk, g.n3), g.zhi) - wk1 + 1;
        const float* kc = ktab + ktab_center(wlev);
        // lanes take the cloud's (ii, jj) pairs and walk its kk planes:
        // each lane forms (m*W(ii))*W(jj) once and the plane loop reads W(kk)
        // as a broadcast.  The pair quotient is exact in float (pairs < 2^11,
        // divisor <= 32).
        const int npair = wdi * wdj;
        const float rdi = s_rcp[wdi];
        const float* wzk = kc + (wk1 - wkz);  // W(kk) of the cloud's planes
        // pair p = (jj-j1)*di + (ii-i1): the lane's first pair by division,
        // the next ones (p += 32) by adding 32 = sj*di + si
        int ci, cj;
        {
          int q0 = (int)(((float)lane + 0.5f) * rdi);
          ci = lane - q0 * wdi;
          cj = q0;
        }
        const int sj = (int)((32.0f + 0.5f) * rdi), si = 32 - sj * wdi;
        for (int pq = lane; pq < npair; pq += 32) {
          const int ii = wi1 + ci, jj = wj1 + cj;
          float bw = __fmul_rn(__fmul_rn(wm, kc[ii - wix]), kc[jj - wjy]);
          double* col = acc + (wk1 - g.zlo) * APLANE + (jj - 1) * AROW + (ii - 1);
#pragma unroll
          for (int q = 0; q < PZ; q++)
            if (q < wdk) atomicAdd(col + q * APLANE, __dmul_rn((double)__fmul_rn(bw, wzk[q]), wc));
          ci += si;
          cj += sj;
          if (ci >= wdi) { ci -= wdi; cj++; }
        }
      }
    }
    vbase += tot;
  }
  __syncthreads();
  const int sidx = W.unit[it.x].x;
  if (sidx < 0) {
    __syncthreads();
    const float den = denbas_lev[g.ir];
    for (int q = threadIdx.x; q < NA * NA * PZ; q += blockDim.x) {
      int i = q % NA, j = (q / NA) % NA, k = g.slab * PZ + q / (NA * NA);
      float v = 0.0f;
      if (i < g.n1 && j < g.n2 && k < g.n3) v = (float)acc[(q / (NA * NA)) * APLANE + j * AROW + i] / den;
      out[q] = v;
    }
  } else {  // one slice of a shared unit
    __syncthreads();
    double* sc = W.scratch + (size_t)sidx * NA * NA * PZ;
    for (int q = threadIdx.x; q < NA * NA * PZ; q += blockDim.x) {
      double a = acc[(q / (NA * NA)) * APLANE + ((q / NA) % NA) * AROW + q % NA];
      if (a != 0.0) atomicAdd(&sc[q], a);
    }
  }
}

// Units shared by several slices: the summed scratch slab to U11.
__global__ void k_patch_finish(DevMesh M, const int32_t* __restrict__ order, const int32_t* __restrict__ multi,
                               const double* __restrict__ scratch, float* __restrict__ u11,
                               const float* __restrict__ denbas_lev) {
  int u = multi[blockIdx.x];
  if (u < 0) return;
  int ip = order[u / NSLAB], slab = u % NSLAB;
  int n1 = M.nx[ip], n2 = M.ny[ip], n3 = M.nz[ip];
  float den = denbas_lev[M.level[ip]];
  const double* sc = scratch + (size_t)blockIdx.x * NA * NA * PZ;
  float* out = u11 + (size_t)ip * NA * NA * NA + (size_t)slab * PZ * NA * NA;
  for (int q = threadIdx.x; q < NA * NA * PZ; q += blockDim.x) {
    int i = q % NA, j = (q / NA) % NA, k = slab * PZ + q / (NA * NA);
    float v = 0.0f;
    if (i < n1 && j < n2 && k < n3) v = (float)sc[q] / den;
    out[q] = v;
  }
}

// Patch order of the deposit: finest level first, table order within a level.
static int patch_order(asohf_ctx* c, const asohf_mesh* mh, int32_t** d_order, DAlloc A = DAlloc{nullptr, false}) {
  int np = 0;
  for (int ir = 1; ir <= mh->nl; ir++) np += mh->npatch[ir];
  std::vector<int32_t> h((size_t)(np > 0 ? np : 1));
  int q = 0;
  for (int ir = mh->nl; ir >= 1; ir--) {
    int first = 0;
    for (int l = 1; l < ir; l++) first += mh->npatch[l];
    for (int p = 0; p < mh->npatch[ir]; p++) h[q++] = first + p;
  }
  const size_t bytes = 4 * (size_t)(np > 0 ? np : 1);
  *d_order = (int32_t*)(A.pool ? A.get(bytes) : arena_alloc(c, bytes));
  if (!*d_order) return ASOHF_ERR_CAPACITY;
  ASOHF_CUDA(cudaMemcpyAsync(*d_order, h.data(), 4 * (size_t)np, cudaMemcpyHostToDevice, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

static float* upload_floats(asohf_ctx* c, const float* h, size_t n, DAlloc A = DAlloc{nullptr, false}) {
  float* d = (float*)(A.pool ? A.get(4 * n) : arena_alloc(c, 4 * n));
  if (d) cudaMemcpyAsync(d, h, 4 * n, cudaMemcpyHostToDevice, c->stream);
  return d;
}

// Output staging: returns a device pointer for `bytes` of output.
static int stage_out(asohf_ctx* c, float* user, size_t bytes, int on_device, float** dev) {
  if (on_device) { *dev = user; return ASOHF_OK; }
  *dev = (float*)arena_alloc(c, bytes);
  return *dev ? ASOHF_OK : ASOHF_ERR_CAPACITY;
}

extern "C" int asohf_density(asohf_ctx* c, int nx, float lado0, float dx, float rote, float rete,
                             const int32_t* npart_esp, const asohf_mesh* mesh, int interp_degree,
                             float* u1, float* u11, int on_device) {
  if (!c || nx <= 0 || !npart_esp || !u1 || (interp_degree != 1 && interp_degree != 2))
    return ASOHF_ERR_INVALID;
  int nl = mesh ? mesh->nl : 0;
  if (nl < 0 || nl > ASOHF_NLEVELS) return ASOHF_ERR_INVALID;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  int64_t n = 0;
  for (int s = 0; s < ASOHF_N_ESP; s++) n += npart_esp[s];
  if (n > c->p.n) return ASOHF_ERR_INVALID;
  int64_t g = (int64_t)nx * nx * nx;
  int np = 0;
  for (int ir = 1; ir <= nl; ir++) np += mesh->npatch[ir];
  if (np > 0 && !u11) return ASOHF_ERR_INVALID;
  const int64_t nall = c->p.n;
  const bool eqmass = c->mmin == c->norma;  // one particle mass in the store
  // the previous call's deferred patch work reads the pools and writes U11
  ASOHF_CHECK(density_settle(c));
  const bool defer = c->density_overlap && on_device && np > 0 && n > 0 && c->dens_stream;
  const DAlloc A{c, defer};
  size_t need = 12 * g + (on_device ? 0 : 4 * g + 4 * (size_t)np * NA * NA * NA) +
                16 * T2COPY + 96 * (size_t)np + 16384 +
                (np ? std::max(bins_bytes(nall, lado0, dx, 2), bins_bytes(nall, lado0, dx, 2, 3)) + 17 * (size_t)nall + unit_list_bytes(NSLAB * np) +
                          8 * NSLAB * (size_t)np : 0);
  ASOHF_CHECK(arena_reserve(c, need));
  if (defer) {  // what the deferred kernels read: mesh, order, bins, staged particles, renorm dims
    const int nbw = (int)lrintf(lado0 / dx);
    const int64_t nb = (nbw + 1) / 2, nbin = nb * nb * nb;
    ASOHF_CHECK(dpool_reserve(c, 0, 16 * T2COPY + 4 * (ASOHF_NLEVELS + 1) + 48 * (size_t)np +
                                        4 * (size_t)(nbin + 1) + 17 * (size_t)nall + 8 * NSLAB * (size_t)np +
                                        16 * 256));
  }
  const float* hk;
  float* dk;
  ASOHF_CHECK(kernel_tables(c, nl, interp_degree, &hk, &dk));
  const float* h0 = hk + ASOHF_NMAX_KERNELS;  // level 0: W(-1), W(0), W(1) at h0[-1..1]
  Terms8 T8;
  for (int q = 0; q < 8; q++) {
    volatile float t = c->norma * h0[q & 1];
    t = t * h0[(q >> 1) & 1];
    t = t * h0[q >> 2];
    T8.t[q] = (double)t;
  }
  // the counting patch kernel: one mass, and every term of every level normal
  bool pd_eq = eqmass;
  for (int ir = 0; ir <= nl; ir++) {
    const float e = hk[(size_t)ir * KW + ASOHF_NMAX_KERNELS + (1 << ir)];
    volatile float t = c->norma * e;
    t = t * e;
    t = t * e;
    if (!(t >= 1.17549435e-38f)) pd_eq = false;
  }
  float* dt2 = nullptr;  // level-2 terms, t[copy][|di|][|dj|][dk], 0 past the cloud
  std::vector<float> ht2;
  if (pd_eq && nl >= 2) {
    const float* k2 = hk + 2 * KW + ASOHF_NMAX_KERNELS;
    ht2.assign(4 * T2COPY, 0.0f);
    for (int cp = 0; cp < 4; cp++)
      for (int a = 0; a <= 4; a++)
        for (int b = 0; b <= 4; b++)
          for (int oz = -4; oz <= 4; oz++) {
            const int e = oz + 7 - cp;
            if (e > 15) continue;
            volatile float t = c->norma * k2[a];
            t = t * k2[b];
            t = t * k2[oz];
            ht2[cp * T2COPY + a * T2A + b * T2R + e] = t;
          }
    dt2 = upload_floats(c, ht2.data(), ht2.size(), A);
    if (!dt2) return ASOHF_ERR_CAPACITY;
  }
  float* du1;
  ASOHF_CHECK(stage_out(c, u1, 4 * g, on_device, &du1));
  const float xl = -lado0 / 2.0f;
  const float denbas = dx * dx * dx * rote * (rete * rete * rete);
  double* acc = (double*)arena_alloc(c, 8 * g);
  int64_t hend[ASOHF_N_ESP];
  int64_t acc_n = 0;
  for (int s = 0; s < ASOHF_N_ESP; s++) { acc_n += npart_esp[s]; hend[s] = acc_n; }
  int64_t* dend = (int64_t*)arena_alloc(c, sizeof(hend));
  int* outside = (int*)arena_alloc(c, 4);
  if (!acc || !dend || !outside) return ASOHF_ERR_CAPACITY;
  ASOHF_CUDA(cudaMemcpyAsync(dend, hend, sizeof(hend), cudaMemcpyHostToDevice, c->stream));
  const float* k0 = dk + ASOHF_NMAX_KERNELS - 1;  // level 0: W(-1), W(0), W(1)
  // the binned copy of the store, which the base grid and the patches read
  const int sub = pd_eq ? 0 : 3;
  Bins B;
  float4* bp = nullptr;
  uint8_t* bs = nullptr;
  if (np > 0 && n > 0) {
    ASOHF_CHECK(build_bins(c, lado0, dx, 2, &B, A, sub));
    bp = (float4*)A.get(16 * (size_t)nall);
    bs = (uint8_t*)A.get((size_t)nall);
    if (!bp || !bs) return ASOHF_ERR_CAPACITY;
    int kt_ = ktime_begin(c, "density_bin_stage");
    k_bin_stage<<<grid_for(nall, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        B.idx, nall, n, c->p.x, c->p.y, c->p.z, c->p.m, c->rows_cur >= 0 ? c->rows[c->rows_cur] : nullptr, dend, bp,
        bs, pd_eq ? 1 : 0);
    ktime_end(c, kt_);
    c->launches++;
  }
  int kt_ = ktime_begin(c, "density_base");
  if (n > 0 && eqmass) {
    int32_t* cnt = (int32_t*)arena_alloc(c, 4 * g);
    if (!cnt) return ASOHF_ERR_CAPACITY;
    ASOHF_CUDA(cudaMemsetAsync(cnt, 0, 4 * g, c->stream));
    ASOHF_CUDA(cudaMemsetAsync(outside, 0, 4, c->stream));
    const bool binned = bp && pd_eq;
    const int64_t nc = binned ? nall : n;
    k_base_counts<<<grid_for(nc, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        c->p.x, c->p.y, c->p.z, binned ? bp : nullptr, nc, nx, xl, dx, cnt, outside);
    const dim3 grid((nx + BS_X - 1) / BS_X, (nx + BS_Y - 1) / BS_Y, (nx + BS_Z - 1) / BS_Z);
    k_base_stencil<<<grid, dim3(BS_X, BS_Y), 0, c->stream>>>(cnt, nx, T8, denbas, outside, acc, du1);
    k_density_base_outliers<<<grid_for(n, 256, c->num_sms * 4), 256, 0, c->stream>>>(
      c->p.x, c->p.y, c->p.z, c->p.m, n, nx, xl, dx, k0, outside, acc);
    k_finish_outliers<<<grid_for(g, 256, c->num_sms * 4), 256, 0, c->stream>>>(outside, acc, g, denbas, du1);
    c->launches += 4;
  } else {
    ASOHF_CUDA(cudaMemsetAsync(acc, 0, 8 * g, c->stream));
    if (n > 0 && bp)
      k_density_base_runs<<<grid_for(nall, 256, c->num_sms * 8), 256, 0, c->stream>>>(bp, bs, nall, nx, xl, dx, k0,
                                                                                      acc);
    else if (n > 0)
      k_density_base_all<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        c->p.x, c->p.y, c->p.z, c->p.m, n, nx, xl, dx, k0, acc);
    k_finish_f64<<<grid_for(g, 256), 256, 0, c->stream>>>(acc, g, denbas, du1);
    c->launches += 1 + (n > 0);
  }
  ktime_end(c, kt_);
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) ASOHF_CUDA(cudaMemcpyAsync(u1, du1, 4 * g, cudaMemcpyDeviceToHost, c->stream));
  if (np > 0) {
    DevMesh M;
    ASOHF_CHECK(upload_mesh(c, mesh, &M, A));
    float hden[ASOHF_NLEVELS + 1];
    for (int ir = 0; ir <= ASOHF_NLEVELS; ir++) {
      float dxpa = dx / powf(2.0f, (float)ir);
      hden[ir] = dxpa * dxpa * dxpa * rote * (rete * rete * rete);
    }
    float* dden = upload_floats(c, hden, ASOHF_NLEVELS + 1, A);
    float* du11;
    ASOHF_CHECK(stage_out(c, u11, 4 * (size_t)np * NA * NA * NA, on_device, &du11));
    int32_t* order = nullptr;
    if (!dden) return ASOHF_ERR_CAPACITY;
    ASOHF_CHECK(patch_order(c, mesh, &order, A));
    if (n > 0) {
      const int nunits = NSLAB * np;
      UnitList U;
      ASOHF_CHECK(unit_list_begin(c, nunits, &U));
      const SliceRule R = pd_eq ? kSliceEq : kSliceAny;
      k_patch_unit_counts<<<(nunits + 7) / 8, 256, 0, c->stream>>>(M, B, order, nunits, dx, pd_eq ? bp : nullptr, bs, R,
                                                                   U.work, U.key, U.unit, U.nm);
      c->launches++;
      // work list: slices of the candidates, the densest units first; in
      // the segment buffers, or density pool 1 when deferred
      ASOHF_CHECK(unit_list_size(c, &U, R));
      const size_t wbytes = unit_work_bytes(U, NA * NA * PZ);
      ASOHF_CHECK(defer ? dpool_reserve(c, 1, wbytes) : seg_reserve(c, wbytes));
      PatchWork W;
      int32_t* dmulti;
      ASOHF_CHECK(unit_list_fill(c, U, NA * NA * PZ,
                                 [&](size_t b) { return defer ? dpool_alloc(c, 1, b) : seg_alloc(c, b); },
                                 [&](size_t b) { return A.get(b); }, &W, &dmulti));
      const size_t smem0 = pd_eq ? sizeof(uint32_t) * CGP * CG * CG + sizeof(float) * 4 * T2COPY
                                 : sizeof(double) * ACC_N;
      const size_t smem = smem0 + sizeof(float) * ktab_size(nl);
      // the limit belongs to the process: the same whatever the levels of a call,
      // so that no other thread's call lowers it before this launch
      ASOHF_CUDA(cudaFuncSetAttribute(pd_eq ? (const void*)k_density_patches_eq : (const void*)k_density_patches,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(smem0 + sizeof(float) * ktab_size(ASOHF_NLEVELS))));
      // deferred: the patch kernels run on the density stream after the
      // staging above, and the call returns without waiting for them
      cudaStream_t ps = c->stream;
      if (defer) {
        ASOHF_CUDA(cudaEventRecord(c->dens_fork, c->stream));
        ASOHF_CUDA(cudaStreamWaitEvent(c->dens_stream, c->dens_fork, 0));
        ps = c->dens_stream;
      }
      int kt_ = ktime_begin(c, "density_patches", ps);
      if (pd_eq)
        k_density_patches_eq<<<(unsigned)U.nitems, PZ_BLOCK, smem, ps>>>(M, B, bp, order, W, dx, dk, c->norma, dt2,
                                                                         du11, dden);
      else
        k_density_patches<<<(unsigned)U.nitems, PZ_BLOCK, smem, ps>>>(M, B, bp, bs, order, W, dx, dk, du11, dden);
      if (U.nmulti) k_patch_finish<<<U.nmulti, 256, 0, ps>>>(M, order, dmulti, W.scratch, du11, dden);
      ktime_end(c, kt_, ps);
      c->launches += 1 + (U.nmulti > 0);
      if (defer) {
        ASOHF_CUDA(cudaEventRecord(c->dens_done, ps));
        c->dens_pending = true;
      }
    } else {  // no particles: empty patches
      ASOHF_CUDA(cudaMemsetAsync(du11, 0, 4 * (size_t)np * NA * NA * NA, c->stream));
    }
    ASOHF_CUDA(cudaGetLastError());
    if (!on_device)
      ASOHF_CUDA(cudaMemcpyAsync(u11, du11, 4 * (size_t)np * NA * NA * NA, cudaMemcpyDeviceToHost, c->stream));
  }
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

// ------------------------------------------------------------ renorm
__global__ void k_scale(float* __restrict__ a, int64_t n, float f) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    a[i] = a[i] / f;
}

__global__ void k_scale_patches(float* __restrict__ u11, const int32_t* __restrict__ dims, int np,
                                float f) {
  int ip = blockIdx.x;
  int n1 = dims[ip], n2 = dims[np + ip], n3 = dims[2 * np + ip];
  float* u = u11 + (size_t)ip * NA * NA * NA;
  for (int q = threadIdx.x; q < NA * NA * NA; q += blockDim.x) {
    int i = q % NA, j = (q / NA) % NA, k = q / (NA * NA);
    if (i < n1 && j < n2 && k < n3) u[q] = u[q] / f;
  }
}

extern "C" int asohf_renorm_density(asohf_ctx* c, int nx, const asohf_mesh* mesh, float fdm,
                                    float* u1, float* u11, int on_device) {
  if (!c || nx <= 0 || !u1) return ASOHF_ERR_INVALID;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  int64_t g = (int64_t)nx * nx * nx;
  int np = 0, nl = mesh ? mesh->nl : 0;
  for (int ir = 1; ir <= nl; ir++) np += mesh->npatch[ir];
  ASOHF_CHECK(arena_reserve(c, (on_device ? 0 : 4 * g + 4 * (size_t)np * NA * NA * NA) + 16 * (size_t)np + 1024));
  float *d1 = u1, *d11 = u11;
  if (!on_device) {
    d1 = (float*)arena_alloc(c, 4 * g);
    ASOHF_CUDA(cudaMemcpyAsync(d1, u1, 4 * g, cudaMemcpyHostToDevice, c->stream));
    if (np) {
      d11 = (float*)arena_alloc(c, 4 * (size_t)np * NA * NA * NA);
      ASOHF_CUDA(cudaMemcpyAsync(d11, u11, 4 * (size_t)np * NA * NA * NA, cudaMemcpyHostToDevice, c->stream));
    }
  }
  k_scale<<<grid_for(g, 256), 256, 0, c->stream>>>(d1, g, fdm);
  c->launches++;
  if (np) {
    int base = mesh->npatch[0];
    std::vector<int32_t> hd(3 * (size_t)np);
    for (int q = 0; q < np; q++) {
      hd[q] = mesh->patchnx[base + q];
      hd[np + q] = mesh->patchny[base + q];
      hd[2 * np + q] = mesh->patchnz[base + q];
    }
    // after a deferred patch deposit the scaling follows it on its stream,
    // with the dimensions in its pool
    const bool deferred = on_device && c->dens_pending;
    int32_t* dd = (int32_t*)(deferred ? dpool_alloc(c, 0, 12 * (size_t)np) : arena_alloc(c, 12 * (size_t)np));
    if (!dd) return ASOHF_ERR_CAPACITY;
    // the dimensions go up on the context stream (a pageable copy on the
    // density stream would make the host wait for the patch kernels)
    ASOHF_CUDA(cudaMemcpyAsync(dd, hd.data(), 12 * (size_t)np, cudaMemcpyHostToDevice, c->stream));
    cudaStream_t ps = c->stream;
    if (deferred) {
      ASOHF_CUDA(cudaEventRecord(c->dens_fork, c->stream));
      ASOHF_CUDA(cudaStreamWaitEvent(c->dens_stream, c->dens_fork, 0));
      ps = c->dens_stream;
    }
    k_scale_patches<<<np, 256, 0, ps>>>(d11, dd, np, fdm);
    c->launches++;
    if (deferred) {
      ASOHF_CUDA(cudaGetLastError());
      ASOHF_CUDA(cudaEventRecord(c->dens_done, ps));
      ASOHF_CUDA(cudaStreamSynchronize(c->stream));  // the base grid; the patches follow on their stream
      return ASOHF_OK;
    }
    ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  }
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) {
    ASOHF_CUDA(cudaMemcpyAsync(u1, d1, 4 * g, cudaMemcpyDeviceToHost, c->stream));
    if (np)
      ASOHF_CUDA(cudaMemcpyAsync(u11, d11, 4 * (size_t)np * NA * NA * NA, cudaMemcpyDeviceToHost, c->stream));
  }
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

// ------------------------------------------------------------ TSC deposit
// Base grid TSC for a batch of particle sets in input order, float32 sums (the
// layer, at the sizes its sort does not cover).
__global__ void k_tsc_base(const float* __restrict__ x, const float* __restrict__ y,
                           const float* __restrict__ z, const float* __restrict__ m, int64_t n_per,
                           int batch, int nx, float xl, float dx, const float* __restrict__ radx,
                           float denbas, float* __restrict__ acc) {
  int64_t ntot = n_per * batch;
  size_t g = (size_t)nx * nx * nx;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < ntot;
       q += (int64_t)gridDim.x * blockDim.x) {
    int b = (int)(q / n_per);
    float xp = x[q], yp = y[q], zp = z[q];
    int ix = tsc_cell(xp, xl, dx, nx), jy = tsc_cell(yp, xl, dx, nx), kz = tsc_cell(zp, xl, dx, nx);
    float wx[3], wy[3], wz[3];
    tsc_weights(xp, radx[ix - 1], radx[ix], radx[ix + 1], dx, wx);
    tsc_weights(yp, radx[jy - 1], radx[jy], radx[jy + 1], dx, wy);
    tsc_weights(zp, radx[kz - 1], radx[kz], radx[kz + 1], dx, wz);
    float mp = denbas == 1.0f ? m[q] : __fdiv_rn(m[q], denbas);  // mass, or mass / DENBAS
    float* a = acc + (size_t)b * g;
#pragma unroll
    for (int kk = -1; kk <= 1; kk++) {
      int k1 = kz + kk;
      if (k1 == nx + 1) k1 = 1;
      if (k1 == 0) k1 = nx;
#pragma unroll
      for (int jj = -1; jj <= 1; jj++) {
        int j1 = jy + jj;
        if (j1 == nx + 1) j1 = 1;
        if (j1 == 0) j1 = nx;
#pragma unroll
        for (int ii = -1; ii <= 1; ii++) {
          int i1 = ix + ii;
          if (i1 == nx + 1) i1 = 1;
          if (i1 == 0) i1 = nx;
          float t = __fmul_rn(__fmul_rn(__fmul_rn(mp, wx[ii + 1]), wy[jj + 1]), wz[kk + 1]);
          atomicAdd(&a[((size_t)(k1 - 1) * nx + (j1 - 1)) * nx + (i1 - 1)], t);
        }
      }
    }
  }
}

// TSC deposits in float64 sums.  A warp holds 32 particles of the binned
// order (one a lane: its cell and 9 weights, the mass already in the x
// weights) in shared memory and then deposits them one cell at a time: lane
// t < 27 takes target cell t of the cloud, adds that target's terms of every
// particle of the warp in the cell and issues one atomic.  A particle a lane
// with 27 atomics each, as before, met itself in a halo's core: the float64
// shared-memory atomic is a compare-and-swap loop, measured 4.7 lane
// operations a clock and SM without conflicts and 0.2 with all lanes on one
// address.
#define TSC_WARP_W 9

__device__ __forceinline__ void tsc_stage(float* w, int lane, float mp, const float* wx, const float* wy,
                                          const float* wz) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    w[lane * TSC_WARP_W + a] = __fmul_rn(mp, wx[a]);
    w[lane * TSC_WARP_W + 3 + a] = wy[a];
    w[lane * TSC_WARP_W + 6 + a] = wz[a];
  }
}

// Sum over the lanes in `grp` of target (i3, j3, k3)'s terms.
__device__ __forceinline__ double tsc_sum(const float* w, unsigned grp, int i3, int j3, int k3) {
  double s = 0.0;
  while (grp) {
    const float* q = w + (__ffs(grp) - 1) * TSC_WARP_W;
    grp &= grp - 1;
    s += (double)__fmul_rn(__fmul_rn(q[i3], q[3 + j3]), q[6 + k3]);
  }
  return s;
}

#define TSC_BLOCK 256
#define TG_BLOCK 64  // k_tsc_base_groups: small sets still reach many SMs

// Periodic base grids of `batch` sets in input order (fewer than 2^31 cells in
// all), m / DENBAS a particle: the runs of k_tsc_base_runs, but the particles of
// a warp that share a cell are found by matching, wherever they sit in it.  The
// atomics on one address are the bound where a set is crowded, so sets of more
// than 65536 particles share them between base_copies() sums of each cell, a
// warp adding to one of them.
//
// Forwards of 160000 particles on 64^3, uniform, in a blob of 1.3 cells, of 0.3
// cells and in one cell: 67, 92, 69 and 53 us; with one sum a cell 63, 163, 116 and
// 62, with 27 atomics a particle 68, 292, 617 and 1324, sorted into float32 sums
// 119, 117, 121 and 122.
__global__ void __launch_bounds__(TG_BLOCK)
k_tsc_base_groups(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                  const float* __restrict__ m, int64_t n_per, int batch, int nx, float xl, float dx,
                  const float* __restrict__ radx, float denbas, int copies, double* __restrict__ acc0) {
  __shared__ float s_w[TG_BLOCK / 32][32 * TSC_WARP_W];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float* w = s_w[threadIdx.x >> 5];
  const int i3 = lane % 3, j3 = (lane / 3) % 3, k3 = min(lane / 9, 2);
  const int64_t n = n_per * batch, g = (int64_t)nx * nx * nx, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  double* acc = acc0 + (warp & (copies - 1)) * batch * g;
  for (int64_t base = warp * 32; base < n; base += nw * 32) {
    const int64_t q = base + lane;
    int ix = 0, jy = 0, kz = 0, b = 0, cell = -1;  // -1: no particle
    if (q < n) {
      const float px = x[q], py = y[q], pz = z[q];
      b = (int)(q / n_per);
      ix = tsc_cell(px, xl, dx, nx);
      jy = tsc_cell(py, xl, dx, nx);
      kz = tsc_cell(pz, xl, dx, nx);
      float wx[3], wy[3], wz[3];
      tsc_weights(px, radx[ix - 1], radx[ix], radx[ix + 1], dx, wx);
      tsc_weights(py, radx[jy - 1], radx[jy], radx[jy + 1], dx, wy);
      tsc_weights(pz, radx[kz - 1], radx[kz], radx[kz + 1], dx, wz);
      tsc_stage(w, lane, denbas == 1.0f ? m[q] : __fdiv_rn(m[q], denbas), wx, wy, wz);
      cell = (int)(b * g) + ((kz - 1) * nx + (jy - 1)) * nx + (ix - 1);
    }
    const unsigned mine = __match_any_sync(FULL, cell);
    unsigned todo = __ballot_sync(FULL, cell >= 0 && lane == __ffs(mine) - 1);
    __syncwarp();
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const unsigned grp = __shfl_sync(FULL, mine, src);
      int i1 = __shfl_sync(FULL, ix, src) + i3 - 1, j1 = __shfl_sync(FULL, jy, src) + j3 - 1,
          k1 = __shfl_sync(FULL, kz, src) + k3 - 1;
      const int bb = __shfl_sync(FULL, b, src);
      if (lane < 27) {
        i1 = i1 == nx + 1 ? 1 : (i1 == 0 ? nx : i1);
        j1 = j1 == nx + 1 ? 1 : (j1 == 0 ? nx : j1);
        k1 = k1 == nx + 1 ? 1 : (k1 == 0 ? nx : k1);
        atomicAdd(&acc[bb * g + ((int64_t)(k1 - 1) * nx + (j1 - 1)) * nx + (i1 - 1)], tsc_sum(w, grp, i3, j3, k3));
      }
    }
    __syncwarp();
  }
}

// Sums of each cell (a power of two) for sets of n_per particles, g cells in all:
// clearing and adding them costs 10 us at 4M cells.
static int base_copies(int64_t n_per, int64_t g) {
  if (n_per <= 65536 || g > (1 << 22)) return 1;
  return g <= (1 << 19) ? 4 : 2;
}

__global__ void k_finish_copies(const double* __restrict__ acc, int64_t g, int copies, float denbas,
                                float* __restrict__ u1) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g;
       c += (int64_t)gridDim.x * blockDim.x) {
    double s = acc[c];
    for (int q = 1; q < copies; q++) s += acc[q * g + c];
    u1[c] = (float)s / denbas;
  }
}

// Periodic base grid, particles in an order that keeps a cell's together.
// Bound by the float64 atomics that remain, one per target and run of a cell:
// 2.1M particles on 128^3 take 0.17 ms with the staging (0.59 ms with one
// atomic per particle and target in file order).
__global__ void __launch_bounds__(TSC_BLOCK)
k_tsc_base_runs(const float4* __restrict__ P, int64_t n, int nx, float xl, float dx, const float* __restrict__ radx,
                double* __restrict__ acc) {
  __shared__ float s_w[TSC_BLOCK / 32][32 * TSC_WARP_W];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float* w = s_w[threadIdx.x >> 5];
  const int i3 = lane % 3, j3 = (lane / 3) % 3, k3 = min(lane / 9, 2);
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n; base += nw * 32) {
    const int64_t q = base + lane;
    int ix = 0, jy = 0, kz = 0;  // 0: no particle
    if (q < n) {
      const float4 p = P[q];
      ix = tsc_cell(p.x, xl, dx, nx);
      jy = tsc_cell(p.y, xl, dx, nx);
      kz = tsc_cell(p.z, xl, dx, nx);
      float wx[3], wy[3], wz[3];
      tsc_weights(p.x, radx[ix - 1], radx[ix], radx[ix + 1], dx, wx);
      tsc_weights(p.y, radx[jy - 1], radx[jy], radx[jy + 1], dx, wy);
      tsc_weights(p.z, radx[kz - 1], radx[kz], radx[kz + 1], dx, wz);
      tsc_stage(w, lane, p.w, wx, wy, wz);
    }
    const int64_t cell = q < n ? ((int64_t)kz * (nx + 2) + jy) * (nx + 2) + ix : -1;
    const int64_t prev = __shfl_up_sync(FULL, cell, 1);
    unsigned heads = __ballot_sync(FULL, q < n && (lane == 0 || prev != cell));
    const unsigned live = __ballot_sync(FULL, q < n);
    __syncwarp();
    while (heads) {
      const int a = __ffs(heads) - 1;
      heads &= heads - 1;
      unsigned grp = live & (FULL << a);
      if (heads) grp &= (1u << (__ffs(heads) - 1)) - 1u;
      int i1 = __shfl_sync(FULL, ix, a) + i3 - 1, j1 = __shfl_sync(FULL, jy, a) + j3 - 1,
          k1 = __shfl_sync(FULL, kz, a) + k3 - 1;
      if (lane < 27) {
        const double s = tsc_sum(w, grp, i3, j3, k3);
        i1 = i1 == nx + 1 ? 1 : (i1 == 0 ? nx : i1);
        j1 = j1 == nx + 1 ? 1 : (j1 == 0 ? nx : j1);
        k1 = k1 == nx + 1 ? 1 : (k1 == 0 ? nx : k1);
        atomicAdd(&acc[((size_t)(k1 - 1) * nx + (j1 - 1)) * nx + (i1 - 1)], s);
      }
    }
    __syncwarp();
  }
}

// Patch TSC (grids.f:1286-1372).  A particle deposits on a patch when it lies
// inside the patch's one-cell buffer.  (The reference also asks PLEV, the
// finest level whose buffered patch holds the particle (grids.f:1121-1152), to
// be at least the patch's own; the buffer is the same box, so a particle
// inside it has such a PLEV and the test never fails.)
// Work unit: TZ planes of one patch in float64 shared memory, its candidates
// in slices as in the DENSITY deposit.  Row and plane strides of 3 and 9
// (mod 16) doubles put the 27 targets of a cloud in different banks.  Bound
// by the warps' per-particle sums and the float64 atomics of single
// particles: 2112 patches over 2.1M particles take 0.63 ms (8.3 ms with one
// CTA per half patch, a particle a lane, read through the bin's index, and
// 1.0 ms more for PLEV).
#define TZ 8
#define TSLAB (NA / TZ)
#define TROW 35
#define TPLANE (NA * TROW + 9)
#define TACC (TZ * TPLANE)

__device__ __forceinline__ void tsc_unit_geo(const DevMesh& M, const Bins& B, int u, float dx, UnitGeo& g) {
  g.ip = u / TSLAB;
  g.slab = u % TSLAB;
  g.n1 = M.nx[g.ip]; g.n2 = M.ny[g.ip]; g.n3 = M.nz[g.ip]; g.ir = M.level[g.ip];
  g.zlo = g.slab * TZ + 1;
  g.zhi = min(g.slab * TZ + TZ, g.n3);
  g.dxpa = dx / exp2f((float)g.ir);
  g.pxl = M.rx[g.ip] - 2.0f * g.dxpa; g.pyl = M.ry[g.ip] - 2.0f * g.dxpa; g.pzl = M.rz[g.ip] - 2.0f * g.dxpa;
  g.pxr = g.pxl + (float)(g.n1 + 2) * g.dxpa;
  g.pyr = g.pyl + (float)(g.n2 + 2) * g.dxpa;
  g.pzr = g.pzl + (float)(g.n3 + 2) * g.dxpa;
  g.bx0 = bin_lo(B, g.pxl); g.bx1 = bin_hi(B, g.pxr);
  g.by0 = bin_lo(B, g.pyl); g.by1 = bin_hi(B, g.pyr);
  // planes zlo..zhi take cells zlo-1..zhi+1, cell k from pzl + k dxpa; half a
  // cell more on each side for the rounding of the quotient
  const float za = fmaxf(g.pzl, g.pzl + ((float)g.zlo - 1.5f) * g.dxpa);
  const float zb = fminf(g.pzr, g.pzl + ((float)g.zhi + 2.5f) * g.dxpa);
  g.bz0 = bin_lo(B, za); g.bz1 = bin_hi(B, zb);
  g.nby = g.by1 - g.by0 + 1;
  g.rows = (g.zlo > g.zhi) ? 0 : g.nby * (g.bz1 - g.bz0 + 1);
}

__global__ void __launch_bounds__(TSC_BLOCK, 3)
k_tsc_patches(DevMesh M, Bins B, const float4* __restrict__ P, PatchWork W, float dx, float* __restrict__ u11,
              const float* __restrict__ denbas_lev) {
  extern __shared__ double acc[];  // TACC doubles
  __shared__ float s_w[TSC_BLOCK / 32][32 * TSC_WARP_W];
  __shared__ int s_lo[PROWS], s_pre[PROWS + 1], s_next;
  const unsigned FULL = 0xffffffffu;
  if (W.past()) return;
  const int2 it = W.items[blockIdx.x];
  UnitGeo g;
  tsc_unit_geo(M, B, it.x, dx, g);
  float* out = u11 + (size_t)g.ip * NA * NA * NA + (size_t)g.slab * TZ * NA * NA;
  if (g.zlo > g.zhi) {  // planes past the patch
    for (int q = threadIdx.x; q < NA * NA * TZ; q += blockDim.x) out[q] = 0.0f;
    return;
  }
  for (int q = threadIdx.x; q < TACC; q += blockDim.x) acc[q] = 0.0;
  const int lane = threadIdx.x & 31;
  float* w = s_w[threadIdx.x >> 5];
  const int i3 = lane % 3, j3 = (lane / 3) % 3, k3 = min(lane / 9, 2);
  const float rx = M.rx[g.ip], ry = M.ry[g.ip], rz = M.rz[g.ip];
  const int slice = W.unit[it.x].y;
  const int64_t v0 = (int64_t)it.y * slice, v1 = v0 + slice;
  int64_t vbase = 0;
  for (int r0 = 0; r0 < g.rows; r0 += PROWS) {
    const int nr = min(PROWS, g.rows - r0);
    __syncthreads();
    stage_rows(B, g, r0, nr, s_lo, s_pre);
    if (threadIdx.x == 0) s_next = (int)(max(v0, vbase) - vbase);
    __syncthreads();
    const int tot = s_pre[nr];
    const int b = (int)(min(v1, vbase + tot) - vbase);
    for (;;) {
      int v = 0;
      if (lane == 0) v = atomicAdd(&s_next, 32);
      v = __shfl_sync(FULL, v, 0);
      if (v >= b) break;
      v += lane;
      int cell = -1;
      if (v < b) {
        const int row = find_row(s_pre, nr, v);
        const float4 p = P[s_lo[row] + (v - s_pre[row])];
        if (g.pxl < p.x && p.x < g.pxr && g.pyl < p.y && p.y < g.pyr && g.pzl < p.z && p.z < g.pzr) {
          const int ix = (int)((p.x - g.pxl) / g.dxpa), jy = (int)((p.y - g.pyl) / g.dxpa),
                    kz = (int)((p.z - g.pzl) / g.dxpa);
          if (kz >= g.zlo - 1 && kz <= g.zhi + 1) {
            // MINIRADX(II) = PATCHRX + (II - 1.5) DXPA
            float wx[3], wy[3], wz[3];
            tsc_weights(p.x, rx + ((float)(ix - 1) - 1.5f) * g.dxpa, rx + ((float)ix - 1.5f) * g.dxpa,
                        rx + ((float)(ix + 1) - 1.5f) * g.dxpa, g.dxpa, wx);
            tsc_weights(p.y, ry + ((float)(jy - 1) - 1.5f) * g.dxpa, ry + ((float)jy - 1.5f) * g.dxpa,
                        ry + ((float)(jy + 1) - 1.5f) * g.dxpa, g.dxpa, wy);
            tsc_weights(p.z, rz + ((float)(kz - 1) - 1.5f) * g.dxpa, rz + ((float)kz - 1.5f) * g.dxpa,
                        rz + ((float)(kz + 1) - 1.5f) * g.dxpa, g.dxpa, wz);
            tsc_stage(w, lane, p.w, wx, wy, wz);
            cell = (kz << 16) | (jy << 8) | ix;  // each 0..NA+2
          }
        }
      }
      const unsigned mine = __match_any_sync(FULL, cell);
      unsigned todo = __ballot_sync(FULL, cell >= 0 && lane == __ffs(mine) - 1);
      __syncwarp();
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned grp = __shfl_sync(FULL, mine, src);
        const int c = __shfl_sync(FULL, cell, src);
        const int i1 = (c & 255) + i3 - 1, j1 = ((c >> 8) & 255) + j3 - 1, k1 = (c >> 16) + k3 - 1;
        if (lane < 27 && i1 > 0 && i1 <= g.n1 && j1 > 0 && j1 <= g.n2 && k1 >= g.zlo && k1 <= g.zhi)
          atomicAdd(&acc[(k1 - g.zlo) * TPLANE + (j1 - 1) * TROW + (i1 - 1)], tsc_sum(w, grp, i3, j3, k3));
      }
      __syncwarp();
    }
    vbase += tot;
  }
  __syncthreads();
  const int sidx = W.unit[it.x].x;
  const float den = denbas_lev[g.ir];
  for (int q = threadIdx.x; q < NA * NA * TZ; q += blockDim.x) {
    const int i = q % NA, j = (q / NA) % NA, k = q / (NA * NA);
    const double a = acc[k * TPLANE + j * TROW + i];
    if (sidx < 0)
      out[q] = i < g.n1 && j < g.n2 && g.slab * TZ + k < g.n3 ? (float)a / den : 0.0f;
    else if (a != 0.0)
      atomicAdd(&W.scratch[(size_t)sidx * NA * NA * TZ + q], a);
  }
}

__global__ void k_tsc_unit_counts(DevMesh M, Bins B, int nunits, float dx, uint32_t* __restrict__ work,
                                  uint32_t* __restrict__ key, int32_t* __restrict__ unit, int32_t* __restrict__ nm) {
  const int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (u >= nunits) return;
  UnitGeo g;
  tsc_unit_geo(M, B, u, dx, g);
  unit_count(B, g, u, lane, [](int) { return 1; }, work, key, unit, nm);
}

// Units shared by several slices: the summed scratch slab to U11.
__global__ void k_tsc_finish(DevMesh M, const int32_t* __restrict__ multi, const double* __restrict__ scratch,
                             float* __restrict__ u11, const float* __restrict__ denbas_lev) {
  const int u = multi[blockIdx.x], ip = u / TSLAB, slab = u % TSLAB;
  if (u < 0) return;
  const int n1 = M.nx[ip], n2 = M.ny[ip], n3 = M.nz[ip];
  const float den = denbas_lev[M.level[ip]];
  const double* sc = scratch + (size_t)blockIdx.x * NA * NA * TZ;
  float* out = u11 + (size_t)ip * NA * NA * NA + (size_t)slab * TZ * NA * NA;
  for (int q = threadIdx.x; q < NA * NA * TZ; q += blockDim.x) {
    const int i = q % NA, j = (q / NA) % NA, k = slab * TZ + q / (NA * NA);
    out[q] = i < n1 && j < n2 && k < n3 ? (float)sc[q] / den : 0.0f;
  }
}

// Without patches a store of up to this many particles deposits in its own
// order: the bins cost more than they save (32768 particles on 64^3 0.054 and
// 0.13 ms, 2.1M on 128^3 0.31 and 0.45, on 256^3 0.57 and 0.62; 6M on 128^3 0.74
// and 0.87, but 1.7 and 0.72, 3.5 and 0.79 where they crowd; 16.8M on 256^3 3.7
// and 3.1).
#define TSC_DIRECT_N (1ll << 21)

extern "C" int asohf_interpolate_density_tsc(asohf_ctx* c, int nx, float lado0, float dx,
                                             const float* radx, float rote, float rete,
                                             const asohf_mesh* mesh, float* u1, float* u11,
                                             int on_device) {
  if (!c || nx <= 0 || !radx || !u1) return ASOHF_ERR_INVALID;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  int64_t n = c->p.n;
  int64_t g = (int64_t)nx * nx * nx;
  int nl = mesh ? mesh->nl : 0;
  int np = 0;
  for (int ir = 1; ir <= nl; ir++) np += mesh->npatch[ir];
  if (np > 0 && !u11) return ASOHF_ERR_INVALID;
  // bins of 2^3 base cells, particles within a bin by eighths of it (its halves,
  // the base cells, without patches): the base grid's cells and the patches'
  // cells to level 2 stay together
  const int bw = 2, sub = np ? 3 : 1, nunits = TSLAB * np;
  const bool direct = np == 0 && n <= TSC_DIRECT_N && g < (1ll << 31);
  const int copies = direct ? base_copies(n, g) : 1;
  size_t need = 8 * g * copies + 4 * g + 4 * (size_t)np * NA * NA * NA + 4 * (nx + 2) + 64 * (size_t)np + 16384 +
                (direct ? 0 : 16 * n + unit_list_bytes(nunits) + bins_bytes(n, lado0, dx, bw, sub));
  ASOHF_CHECK(arena_reserve(c, need));
  float* dradx = upload_floats(c, radx, nx + 2);
  double* acc = (double*)arena_alloc(c, 8 * g * copies);
  float4* bp = direct ? nullptr : (float4*)arena_alloc(c, 16 * n + 16);
  float* du1;
  ASOHF_CHECK(stage_out(c, u1, 4 * g, on_device, &du1));
  if (!dradx || !acc || (!direct && !bp)) return ASOHF_ERR_CAPACITY;
  ASOHF_CUDA(cudaMemsetAsync(acc, 0, 8 * g * copies, c->stream));
  float xl = -lado0 / 2.0f;
  Bins B;
  if (n > 0 && direct) {
    int kt_ = ktime_begin(c, "tsc_base");
    k_tsc_base_groups<<<grid_for(n, TG_BLOCK, c->num_sms * 16), TG_BLOCK, 0, c->stream>>>(
        c->p.x, c->p.y, c->p.z, c->p.m, n, 1, nx, xl, dx, dradx, 1.0f, copies, acc);
    ktime_end(c, kt_);
    c->launches++;
  } else if (n > 0) {
    ASOHF_CHECK(build_bins(c, lado0, dx, bw, &B, DAlloc{nullptr, false}, sub));
    int kt_ = ktime_begin(c, "tsc_base");
    k_bin_stage<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        B.idx, n, n, c->p.x, c->p.y, c->p.z, c->p.m, c->rows_cur >= 0 ? c->rows[c->rows_cur] : nullptr, nullptr, bp,
        nullptr, 0);
    k_tsc_base_runs<<<grid_for(n, TSC_BLOCK, c->num_sms * 8), TSC_BLOCK, 0, c->stream>>>(bp, n, nx, xl, dx, dradx,
                                                                                         acc);
    ktime_end(c, kt_);
    c->launches += 2;
  }
  float denbas = dx * dx * dx * rote * (rete * rete * rete);
  k_finish_copies<<<grid_for(g, 256), 256, 0, c->stream>>>(acc, g, copies, denbas, du1);
  c->launches++;
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) ASOHF_CUDA(cudaMemcpyAsync(u1, du1, 4 * g, cudaMemcpyDeviceToHost, c->stream));
  if (np > 0) {
    float* du11;
    ASOHF_CHECK(stage_out(c, u11, 4 * (size_t)np * NA * NA * NA, on_device, &du11));
    DevMesh M;
    ASOHF_CHECK(upload_mesh(c, mesh, &M));
    if (n > 0) {
      float hden[ASOHF_NLEVELS + 1];
      for (int ir = 0; ir <= ASOHF_NLEVELS; ir++) {
        float dxpa = dx / powf(2.0f, (float)ir);
        hden[ir] = dxpa * dxpa * dxpa * rote * (rete * rete * rete);
      }
      float* dden = upload_floats(c, hden, ASOHF_NLEVELS + 1);
      if (!dden) return ASOHF_ERR_CAPACITY;
      UnitList U;
      ASOHF_CHECK(unit_list_begin(c, nunits, &U));
      k_tsc_unit_counts<<<(nunits + 7) / 8, 256, 0, c->stream>>>(M, B, nunits, dx, U.work, U.key, U.unit, U.nm);
      c->launches++;
      ASOHF_CHECK(unit_list_size(c, &U, kSliceUnits));
      ASOHF_CHECK(seg_reserve(c, unit_work_bytes(U, NA * NA * TZ)));
      PatchWork W;
      int32_t* multi;
      ASOHF_CHECK(unit_list_fill(c, U, NA * NA * TZ, [&](size_t b) { return seg_alloc(c, b); },
                                 [&](size_t b) { return arena_alloc(c, b); }, &W, &multi));
      const size_t smem = sizeof(double) * TACC;
      ASOHF_CUDA(cudaFuncSetAttribute(k_tsc_patches, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      int kt_ = ktime_begin(c, "tsc_patches");
      k_tsc_patches<<<(unsigned)U.nitems, TSC_BLOCK, smem, c->stream>>>(M, B, bp, W, dx, du11, dden);
      if (U.nmulti) k_tsc_finish<<<U.nmulti, 256, 0, c->stream>>>(M, multi, W.scratch, du11, dden);
      ktime_end(c, kt_);
      c->launches += 1 + (U.nmulti > 0);
      ASOHF_CUDA(cudaGetLastError());
    } else {  // no particles: empty patches
      ASOHF_CUDA(cudaMemsetAsync(du11, 0, 4 * (size_t)np * NA * NA * NA, c->stream));
    }
    if (!on_device)
      ASOHF_CUDA(cudaMemcpyAsync(u11, du11, 4 * (size_t)np * NA * NA * NA, cudaMemcpyDeviceToHost, c->stream));
  }
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

// exported for poisson.cu (batched forward deposit of m / denbas)
int tsc_base_batched_f32(asohf_ctx* c, int nx, float xl, float dx, const float* dradx, int batch,
                         int64_t n_per, const float* x, const float* y, const float* z,
                         const float* m, float denbas, float* acc) {
  int64_t n = n_per * batch;
  if (n > 0) {
    {
      int kt_ = ktime_begin(c, "tsc_base_batched");
      k_tsc_base<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(x, y, z, m, n_per, batch, nx, xl, dx,
                                                                           dradx, denbas, acc);
      ktime_end(c, kt_);
    }
    c->launches++;
  }
  ASOHF_CUDA(cudaGetLastError());
  return ASOHF_OK;
}

// the same in float64 sums (tsc_base_f64_bytes of scratch), rounded into rho
size_t tsc_base_f64_bytes(int64_t n_per, int64_t g) { return 8 * (size_t)g * base_copies(n_per, g); }

int tsc_base_batched_f64(asohf_ctx* c, int nx, float xl, float dx, const float* dradx, int batch,
                         int64_t n_per, const float* x, const float* y, const float* z,
                         const float* m, float denbas, double* acc, float* rho) {
  const int64_t n = n_per * batch, g = (int64_t)nx * nx * nx * batch;
  const int copies = base_copies(n_per, g);
  ASOHF_CUDA(cudaMemsetAsync(acc, 0, tsc_base_f64_bytes(n_per, g), c->stream));
  int kt_ = ktime_begin(c, "tsc_base_batched");
  if (n > 0) {
    k_tsc_base_groups<<<grid_for(n, TG_BLOCK, c->num_sms * 16), TG_BLOCK, 0, c->stream>>>(
        x, y, z, m, n_per, batch, nx, xl, dx, dradx, denbas, copies, acc);
    c->launches++;
  }
  k_finish_copies<<<grid_for(g, 256), 256, 0, c->stream>>>(acc, g, copies, 1.0f, rho);
  c->launches++;
  ktime_end(c, kt_);
  ASOHF_CUDA(cudaGetLastError());
  return ASOHF_OK;
}

// ------------------------------------------------------------ CREATE_MESH particle counts
// The two counting loops of CREATE_MESH (grids.f:107-143 for the base grid,
// grids.f:357-380 for the patches of one level): NGP cell counts in which a
// particle weighs 1 when its species level PLEV is at most the level being
// refined (0 for the base grid) and REFINE_THR otherwise, then zero within
// BOR (BORAMR) cells of the faces.  PLEV(I) is the species whose index range
// (NPART_ESP, store order) holds I, and 0 past the last range (grids.f:83-91).
// The patch placement that consumes the counts is sequential and stays with
// the caller.

struct EspEnds {
  int64_t e[ASOHF_N_ESP];  // cumulative ends of the species ranges
};

__device__ __forceinline__ int plev_of(int64_t i, const EspEnds& E) {
  for (int s = 0; s < ASOHF_N_ESP; s++)
    if (i < E.e[s]) return s;
  return 0;
}

__global__ void k_mesh_base_counts(const float* __restrict__ x, const float* __restrict__ y,
                                   const float* __restrict__ z, int64_t n, int nx, float xl, float dx,
                                   int refine_thr, EspEnds E, int32_t* __restrict__ cnt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    // IX = INT((RXPA-XL)/DX)+1 clamped to 1..NX (a NaN offset counts as below)
    int c3[3];
    const float v3[3] = {x[i], y[i], z[i]};
    for (int a = 0; a < 3; a++) {
      const float v = __fdiv_rn(__fsub_rn(v3[a], xl), dx);
      c3[a] = v >= (float)nx ? nx : (v >= 1.0f ? (int)v + 1 : 1);
    }
    const int w = plev_of(i, E) == 0 ? 1 : refine_thr;
    atomicAdd(&cnt[((int64_t)(c3[2] - 1) * nx + (c3[1] - 1)) * nx + (c3[0] - 1)], w);
  }
}

__global__ void k_mesh_border(int32_t* __restrict__ cnt, int nx, int bor) {
  const int64_t g = (int64_t)nx * nx * nx;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < g; q += (int64_t)gridDim.x * blockDim.x) {
    const int ix = (int)(q % nx) + 1, jy = (int)((q / nx) % nx) + 1, kz = (int)(q / ((int64_t)nx * nx)) + 1;
    if (ix <= bor || ix >= nx - bor + 1 || jy <= bor || jy >= nx - bor + 1 || kz <= bor || kz >= nx - bor + 1)
      cnt[q] = 0;
  }
}

// Patches of the level in units of MZ planes: int32 counts in shared memory,
// candidates from the binned store (x, y, z, weight) over the bins covering the
// unit widened by two fine cells (a superset of the particles the FLOOR test
// keeps, for cells wider than the float spacing of the coordinates), in slices
// as in the deposits; the slices of a unit add to the output, cleared before.
// Bound by the candidate scan: 2500 patches of 4.1M particles take 0.38 ms (1.29
// ms with one CTA a patch reading positions through the bin's index).
#define MZ 8
#define MSLAB (NA / MZ)

struct MeshPatches {
  const int32_t* n;  // PATCHNX, Y, Z
  const float* r;    // PATCHRX, Y, Z
  int np, boramr;
  float dxpa;
};

__device__ __forceinline__ void mesh_unit_geo(const MeshPatches& M, const Bins& B, int u, UnitGeo& g) {
  g.ip = u / MSLAB;
  g.slab = u % MSLAB;
  g.n1 = M.n[g.ip]; g.n2 = M.n[M.np + g.ip]; g.n3 = M.n[2 * M.np + g.ip];
  g.zlo = g.slab * MZ;  // 0-based planes zlo .. zhi
  g.zhi = min(g.zlo + MZ, g.n3) - 1;
  g.dxpa = M.dxpa;
  // XL = PATCHRX - DXPA (grids.f:358-360)
  g.xlfix = __fsub_rn(M.r[g.ip], M.dxpa);
  g.ylfix = __fsub_rn(M.r[M.np + g.ip], M.dxpa);
  g.zlfix = __fsub_rn(M.r[2 * M.np + g.ip], M.dxpa);
  const float pad = 2.0f * M.dxpa;
  g.bx0 = bin_lo(B, g.xlfix - pad);
  g.bx1 = bin_hi(B, g.xlfix + (float)(g.n1 + 2) * M.dxpa);
  g.by0 = bin_lo(B, g.ylfix - pad);
  g.by1 = bin_hi(B, g.ylfix + (float)(g.n2 + 2) * M.dxpa);
  g.bz0 = bin_lo(B, g.zlfix + (float)(g.zlo - 2) * M.dxpa);
  g.bz1 = bin_hi(B, g.zlfix + (float)(g.zhi + 3) * M.dxpa);
  g.nby = g.by1 - g.by0 + 1;
  g.rows = g.zlo > g.zhi ? 0 : g.nby * (g.bz1 - g.bz0 + 1);
}

__global__ void k_mesh_unit_counts(MeshPatches M, Bins B, int nunits, uint32_t* __restrict__ work,
                                   uint32_t* __restrict__ key, int32_t* __restrict__ unit, int32_t* __restrict__ nm) {
  const int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (u >= nunits) return;
  UnitGeo g;
  mesh_unit_geo(M, B, u, g);
  unit_count(B, g, u, lane, [](int) { return 1; }, work, key, unit, nm);
}

// The store in bin order with each particle's weight on the level.
__global__ void k_mesh_stage(const int32_t* __restrict__ idx, int64_t n, const float* __restrict__ x,
                             const float* __restrict__ y, const float* __restrict__ z,
                             const float4* __restrict__ rows, int irpa, int refine_thr, EspEnds E,
                             float4* __restrict__ P) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int p = idx[t];
    float4 v = rows ? rows[2 * (int64_t)p] : make_float4(x[p], y[p], z[p], 0.f);
    v.w = __int_as_float(plev_of(p, E) <= irpa ? 1 : refine_thr);
    P[t] = v;
  }
}

__global__ void __launch_bounds__(256)
k_mesh_patch_counts(MeshPatches M, Bins B, const float4* __restrict__ P, PatchWork W, int32_t* __restrict__ out) {
  __shared__ int32_t s_cnt[MZ * NA * NA];
  __shared__ int s_lo[PROWS], s_pre[PROWS + 1];
  if (W.past()) return;
  const int2 it = W.items[blockIdx.x];
  UnitGeo g;
  mesh_unit_geo(M, B, it.x, g);
  for (int q = threadIdx.x; q < MZ * NA * NA; q += blockDim.x) s_cnt[q] = 0;
  const int slice = W.unit[it.x].y;
  const int64_t v0 = (int64_t)it.y * slice, v1 = v0 + slice;
  int64_t vbase = 0;
  for (int r0 = 0; r0 < g.rows; r0 += PROWS) {
    const int nr = min(PROWS, g.rows - r0);
    __syncthreads();
    stage_rows(B, g, r0, nr, s_lo, s_pre);
    __syncthreads();
    const int tot = s_pre[nr];
    const int a = (int)(max(v0, vbase) - vbase), b = (int)(min(v1, vbase + tot) - vbase);
    for (int v = a + threadIdx.x; v < b; v += blockDim.x) {
      const int row = find_row(s_pre, nr, v);
      const float4 p = P[s_lo[row] + (v - s_pre[row])];
      // IX = FLOOR((RXPA-XL)/DXPA)+1 kept when 1 <= IX <= N1
      const float vz = __fdiv_rn(__fsub_rn(p.z, g.zlfix), g.dxpa);
      if (!(vz >= 0.0f && vz < (float)g.n3) || (int)vz < g.zlo || (int)vz > g.zhi) continue;
      const float vx = __fdiv_rn(__fsub_rn(p.x, g.xlfix), g.dxpa);
      if (!(vx >= 0.0f && vx < (float)g.n1)) continue;
      const float vy = __fdiv_rn(__fsub_rn(p.y, g.ylfix), g.dxpa);
      if (!(vy >= 0.0f && vy < (float)g.n2)) continue;
      atomicAdd(&s_cnt[(((int)vz - g.zlo) * NA + (int)vy) * NA + (int)vx], __float_as_int(p.w));
    }
    vbase += tot;
  }
  __syncthreads();
  const bool shared = W.unit[it.x].x >= 0;
  const int bor = M.boramr;
  int32_t* o = out + ((size_t)g.ip * NA + g.zlo) * NA * NA;
  for (int q = threadIdx.x; q < MZ * NA * NA; q += blockDim.x) {
    const int ix = q % NA + 1, jy = (q / NA) % NA + 1, kz = g.zlo + q / (NA * NA) + 1;
    int v = s_cnt[q];
    if (ix > g.n1 || jy > g.n2 || kz > g.n3 || ix <= bor || ix >= g.n1 - bor + 1 || jy <= bor ||
        jy >= g.n2 - bor + 1 || kz <= bor || kz >= g.n3 - bor + 1)
      v = 0;
    if (!shared) o[q] = v;
    else if (v) atomicAdd(&o[q], v);
  }
}

// Clears the output of the units that several slices share.
__global__ void k_mesh_clear(const int32_t* __restrict__ multi, int32_t* __restrict__ out) {
  if (multi[blockIdx.x] < 0) return;
  int32_t* o = out + (size_t)multi[blockIdx.x] * MZ * NA * NA;
  for (int q = threadIdx.x; q < MZ * NA * NA; q += blockDim.x) o[q] = 0;
}

static int esp_ends(const int32_t* npart_esp, EspEnds* E) {
  int64_t acc = 0;
  for (int s = 0; s < ASOHF_N_ESP; s++) {
    if (npart_esp[s] < 0) return ASOHF_ERR_INVALID;
    acc += npart_esp[s];
    E->e[s] = acc;
  }
  return ASOHF_OK;
}

extern "C" int asohf_mesh_base_counts(asohf_ctx* c, int nx, float dx, int refine_thr, int bor,
                                      const int32_t* npart_esp, int32_t* cr0, int on_device) {
  if (!c || nx <= 0 || !npart_esp || !cr0) return ASOHF_ERR_INVALID;
  EspEnds E;
  ASOHF_CHECK(esp_ends(npart_esp, &E));
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  const int64_t g = (int64_t)nx * nx * nx, n = c->p.n;
  ASOHF_CHECK(arena_reserve(c, 4 * (size_t)g + 4096));
  int32_t* d = on_device ? cr0 : (int32_t*)arena_alloc(c, 4 * (size_t)g);
  if (!d) return ASOHF_ERR_CAPACITY;
  ASOHF_CUDA(cudaMemsetAsync(d, 0, 4 * (size_t)g, c->stream));
  const float xl = -((float)nx * dx / 2.0f);  // XL = -NX*DX/2.
  int kt_ = ktime_begin(c, "mesh_base_counts");
  if (n > 0) {
    k_mesh_base_counts<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(c->p.x, c->p.y, c->p.z, n, nx, xl,
                                                                                  dx, refine_thr, E, d);
    c->launches++;
  }
  k_mesh_border<<<grid_for(g, 256), 256, 0, c->stream>>>(d, nx, bor);
  c->launches++;
  ktime_end(c, kt_);
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) ASOHF_CUDA(cudaMemcpyAsync(cr0, d, 4 * (size_t)g, cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

extern "C" int asohf_mesh_patch_counts(asohf_ctx* c, int nx, float lado0, float dx, int irpa, int refine_thr,
                                       int boramr, const int32_t* npart_esp, int npatch, const int32_t* patchnx,
                                       const int32_t* patchny, const int32_t* patchnz, const float* patchrx,
                                       const float* patchry, const float* patchrz, int32_t* cr01, int on_device) {
  if (!c || nx <= 0 || irpa < 1 || npatch < 0 || !npart_esp || (npatch > 0 && (!patchnx || !patchny || !patchnz ||
      !patchrx || !patchry || !patchrz || !cr01)))
    return ASOHF_ERR_INVALID;
  EspEnds E;
  ASOHF_CHECK(esp_ends(npart_esp, &E));
  for (int q = 0; q < npatch; q++)
    if (patchnx[q] < 1 || patchnx[q] > NA || patchny[q] < 1 || patchny[q] > NA || patchnz[q] < 1 || patchnz[q] > NA)
      return ASOHF_ERR_INVALID;
  if (npatch == 0) return ASOHF_OK;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  const int64_t n = c->p.n;
  const size_t outb = 4 * (size_t)npatch * NA * NA * NA;
  const int nunits = MSLAB * npatch;
  ASOHF_CHECK(arena_reserve(c, (on_device ? 0 : outb) + (24 + 8 * MSLAB) * (size_t)npatch + 16 * (size_t)n +
                                   unit_list_bytes(nunits) + bins_bytes(n, lado0, dx, 2) + 16384));
  int32_t* pn = (int32_t*)arena_alloc(c, 12 * (size_t)npatch);
  float* pr = (float*)arena_alloc(c, 12 * (size_t)npatch);
  int32_t* d = on_device ? cr01 : (int32_t*)arena_alloc(c, outb);
  if (!pn || !pr || !d) return ASOHF_ERR_CAPACITY;
  const int32_t* hn[3] = {patchnx, patchny, patchnz};
  const float* hr[3] = {patchrx, patchry, patchrz};
  for (int a = 0; a < 3; a++) {
    ASOHF_CUDA(cudaMemcpyAsync(pn + (size_t)a * npatch, hn[a], 4 * (size_t)npatch, cudaMemcpyHostToDevice, c->stream));
    ASOHF_CUDA(cudaMemcpyAsync(pr + (size_t)a * npatch, hr[a], 4 * (size_t)npatch, cudaMemcpyHostToDevice, c->stream));
  }
  Bins B;
  ASOHF_CHECK(build_bins(c, lado0, dx, 2, &B));
  const float dxpa = ldexpf(dx, -irpa);  // DX/(2.0**IRPA), exact
  float4* bp = (float4*)arena_alloc(c, 16 * (size_t)n + 16);
  if (!bp) return ASOHF_ERR_CAPACITY;
  const MeshPatches M{pn, pr, npatch, boramr, dxpa};
  UnitList U;
  ASOHF_CHECK(unit_list_begin(c, nunits, &U));
  int kt_ = ktime_begin(c, "mesh_patch_counts");
  if (n > 0)
    k_mesh_stage<<<grid_for(n, 256, c->num_sms * 16), 256, 0, c->stream>>>(
        B.idx, n, c->p.x, c->p.y, c->p.z, c->rows_cur >= 0 ? c->rows[c->rows_cur] : nullptr, irpa, refine_thr, E, bp);
  k_mesh_unit_counts<<<(nunits + 7) / 8, 256, 0, c->stream>>>(M, B, nunits, U.work, U.key, U.unit, U.nm);
  ASOHF_CHECK(unit_list_size(c, &U, kSliceUnits));
  ASOHF_CHECK(seg_reserve(c, unit_work_bytes(U, 0)));
  PatchWork W;
  int32_t* multi;
  ASOHF_CHECK(unit_list_fill(c, U, 0, [&](size_t b) { return seg_alloc(c, b); },
                             [&](size_t b) { return arena_alloc(c, b); }, &W, &multi));
  if (U.nmulti) k_mesh_clear<<<U.nmulti, 256, 0, c->stream>>>(multi, d);
  k_mesh_patch_counts<<<(unsigned)U.nitems, 256, 0, c->stream>>>(M, B, bp, W, d);
  c->launches += 2 + (n > 0) + (U.nmulti > 0);
  ktime_end(c, kt_);
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) ASOHF_CUDA(cudaMemcpyAsync(cr01, d, outb, cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

// ------------------------------------------------------------ VEINSGRID_REDUCED
// grids.f:1771-2073.  Patch I (in order) marks the cells of each neighbour J
// that face an unmarked cell of I; a row reads only I's marks and writes
// only its neighbours', and the neighbour relation (intersecting cell boxes
// on the level's grid) is symmetric.  So rows whose patches do not
// intersect commute, and the rows are replayed in waves: a row's wave is
// one past the latest wave of its lower-index neighbours, and one launch
// takes a wave with one CTA per row.  The result equals the sequential one.

__device__ __forceinline__ int veins_int(float v) { return (int)__fadd_rn(v, 0.5f); }  // INT(v+0.5)

// Lower cell of each patch on the level's grid (IG1, JG1, KG1).
__global__ void k_veins_box(const int32_t* __restrict__ pn, const float* __restrict__ pr, int np, float dxpa,
                            float fix, int32_t* __restrict__ g1) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= 3 * np) return;
  const float r1 = __fsub_rn(pr[q], __fmul_rn(0.5f, dxpa));
  g1[q] = veins_int(__fdiv_rn(__fsub_rn(r1, fix), dxpa)) + 1;
}

__device__ __forceinline__ bool veins_meet(const int32_t* g1, const int32_t* pn, int np, int i, int j) {
  bool ok = true;
  for (int a = 0; a < 3; a++) {
    const int gi = g1[a * np + i], gj = g1[a * np + j];
    ok = ok && gi <= gj + pn[a * np + j] - 1 && gj <= gi + pn[a * np + i] - 1;
  }
  return ok;
}

// Neighbours of each patch, in index order: counts (fill == nullptr) or the
// list.  One warp per patch, 32 partners a step.
__global__ void k_veins_neighbours(const int32_t* __restrict__ g1, const int32_t* __restrict__ pn, int np,
                                   int32_t* __restrict__ cnt, const int32_t* __restrict__ off,
                                   int32_t* __restrict__ fill) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= np) return;
  int k = 0;
  for (int j0 = 0; j0 < np; j0 += 32) {
    const int j = j0 + lane;
    const bool in = j < np && j != i && veins_meet(g1, pn, np, i, j);
    const unsigned msk = __ballot_sync(0xffffffffu, in);
    if (fill && in) fill[off[i] + k + __popc(msk & ((1u << lane) - 1u))] = j;
    k += __popc(msk);
  }
  if (!fill && lane == 0) cnt[i] = k;
}

// The overlap corners of one axis (the four cases of grids.f:1965-2026).
__device__ __forceinline__ void veins_axis_d(float r1, float r2, float rr1, float rr2, float dxpa, int n, int nn,
                                             int* c1, int* c2, int* cc1, int* cc2) {
  if (rr1 >= r1 && rr2 <= r2) {
    *c1 = veins_int(__fdiv_rn(__fsub_rn(rr1, r1), dxpa)) + 1;
    *c2 = veins_int(__fdiv_rn(__fsub_rn(rr2, r1), dxpa)) + 1;
    *cc1 = 1;
    *cc2 = nn;
  }
  if (rr1 >= r1 && rr2 > r2) {
    *c1 = veins_int(__fdiv_rn(__fsub_rn(rr1, r1), dxpa)) + 1;
    *c2 = n;
    *cc1 = 1;
    *cc2 = veins_int(__fdiv_rn(__fsub_rn(r2, rr1), dxpa)) + 1;
  }
  if (rr2 <= r2 && rr1 < r1) {
    *c1 = 1;
    *c2 = veins_int(__fdiv_rn(__fsub_rn(rr2, r1), dxpa)) + 1;
    *cc1 = veins_int(__fdiv_rn(__fsub_rn(r1, rr1), dxpa)) + 1;
    *cc2 = nn;
  }
  if (rr1 < r1 && rr2 > r2) {
    *c1 = 1;
    *c2 = n;
    *cc1 = veins_int(__fdiv_rn(__fsub_rn(r1, rr1), dxpa)) + 1;
    *cc2 = veins_int(__fdiv_rn(__fsub_rn(r2, rr1), dxpa)) + 1;
  }
}

// A wave's rows, patch I against each neighbour J: one CTA per (J, row).  The
// pairs of a wave do not depend on one another: a row reads its own patch's
// marks, which no row of its wave writes.  (One CTA per row walked its
// neighbours in turn: 2500 level-1 patches of a 160^3 box 1.17 ms, so 0.22.)
__global__ void __launch_bounds__(256) k_veins_rows(const int32_t* __restrict__ rows, const int32_t* __restrict__ off,
                                                    const int32_t* __restrict__ nb, const int32_t* __restrict__ pn,
                                                    const float* __restrict__ pr, int np, float dxpa,
                                                    uint8_t* __restrict__ solap, int32_t* __restrict__ cr01,
                                                    int32_t* __restrict__ conta11) {
  const int i = rows[blockIdx.x];
  const size_t pc = (size_t)NA * NA * NA;
  float r1[3], r2[3];
  int n[3];
  for (int a = 0; a < 3; a++) {
    n[a] = pn[a * np + i];
    r1[a] = __fsub_rn(pr[a * np + i], __fmul_rn(0.5f, dxpa));
    r2[a] = __fadd_rn(r1[a], __fmul_rn((float)(n[a] - 1), dxpa));
  }
  for (int k = off[i] + blockIdx.y; k < off[i + 1]; k += gridDim.y) {
    const int j = nb[k];
    int c1[3], c2[3], cc1[3], cc2[3], e[3];
    for (int a = 0; a < 3; a++) {
      const int nn = pn[a * np + j];
      const float rr1 = __fsub_rn(pr[a * np + j], __fmul_rn(0.5f, dxpa));
      const float rr2 = __fadd_rn(rr1, __fmul_rn((float)(nn - 1), dxpa));
      c1[a] = c2[a] = cc1[a] = cc2[a] = 0;
      veins_axis_d(r1[a], r2[a], rr1, rr2, dxpa, n[a], nn, &c1[a], &c2[a], &cc1[a], &cc2[a]);
      e[a] = cc2[a] - cc1[a] + 1;
    }
    const int prod = e[2] * e[1] * e[0];
    const float ov = __fdiv_rn(__fdiv_rn(__fdiv_rn(fabsf((float)prod), (float)pn[j]), (float)pn[np + j]),
                               (float)pn[2 * np + j]);
    if (!(ov > 0.1f) || e[0] <= 0 || e[1] <= 0 || e[2] <= 0) continue;
    const int ncell = e[0] * e[1] * e[2];
    for (int q = threadIdx.x; q < ncell; q += blockDim.x) {
      const int ii = cc1[0] + q % e[0], jj = cc1[1] + (q / e[0]) % e[1], kk = cc1[2] + q / (e[0] * e[1]);
      const int ix = ii - cc1[0] + c1[0], jy = jj - cc1[1] + c1[1], kz = kk - cc1[2] + c1[2];
      if (ii < 1 || ii > NA || jj < 1 || jj > NA || kk < 1 || kk > NA || ix < 1 || ix > NA || jy < 1 || jy > NA ||
          kz < 1 || kz > NA)
        continue;  // outside the NAMRX^3 arrays
      const size_t qi = (size_t)i * pc + ((size_t)(kz - 1) * NA + (jy - 1)) * NA + (ix - 1);
      const size_t qj = (size_t)j * pc + ((size_t)(kk - 1) * NA + (jj - 1)) * NA + (ii - 1);
      if (solap[qi] == 0) {
        solap[qj] = 1;
        cr01[qj] = 0;
        if (conta11) conta11[qj] = 0;
      }
    }
  }
}

extern "C" int asohf_veinsgrid_reduced(asohf_ctx* c, int ir, float dx, float radx1, int npatch,
                                       const int32_t* patchnx, const int32_t* patchny, const int32_t* patchnz,
                                       const float* patchrx, const float* patchry, const float* patchrz,
                                       int max_neighbours, int32_t* cr01, int32_t* conta11, int on_device) {
  if (!c || ir < 1 || npatch < 0 || max_neighbours < 0 ||
      (npatch > 0 && (!patchnx || !patchny || !patchnz || !patchrx || !patchry || !patchrz || !cr01)))
    return ASOHF_ERR_INVALID;
  for (int q = 0; q < npatch; q++)
    if (patchnx[q] < 1 || patchnx[q] > NA || patchny[q] < 1 || patchny[q] > NA || patchnz[q] < 1 || patchnz[q] > NA)
      return ASOHF_ERR_INVALID;
  if (npatch == 0) return ASOHF_OK;
  ASOHF_CUDA(cudaSetDevice(c->device));
  arena_reset(c);
  const int np = npatch;
  const size_t pc = (size_t)NA * NA * NA;
  size_t tb = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tb, (int32_t*)nullptr, (int32_t*)nullptr, np + 1);
  const size_t host_b = on_device ? 0 : 4 * pc * (size_t)np * (conta11 ? 2 : 1);
  ASOHF_CHECK(arena_reserve(c, host_b + pc * (size_t)np + 48 * (size_t)np + tb + 16 * 256 + 4096));
  int32_t* pn = (int32_t*)arena_alloc(c, 12 * (size_t)np);
  float* pr = (float*)arena_alloc(c, 12 * (size_t)np);
  int32_t* g1 = (int32_t*)arena_alloc(c, 12 * (size_t)np);
  int32_t* cnt = (int32_t*)arena_alloc(c, 4 * (size_t)np + 4);
  int32_t* off = (int32_t*)arena_alloc(c, 4 * (size_t)np + 4);
  int32_t* rows = (int32_t*)arena_alloc(c, 4 * (size_t)np);
  void* tmp = arena_alloc(c, tb);
  uint8_t* solap = (uint8_t*)arena_alloc(c, pc * (size_t)np);
  int32_t* dcr = on_device ? cr01 : (int32_t*)arena_alloc(c, 4 * pc * (size_t)np);
  int32_t* dct = (!conta11 || on_device) ? conta11 : (int32_t*)arena_alloc(c, 4 * pc * (size_t)np);
  if (!pn || !pr || !g1 || !cnt || !off || !rows || !tmp || !solap || !dcr || (conta11 && !dct))
    return ASOHF_ERR_CAPACITY;
  const int32_t* hn[3] = {patchnx, patchny, patchnz};
  const float* hr[3] = {patchrx, patchry, patchrz};
  for (int a = 0; a < 3; a++) {
    ASOHF_CUDA(cudaMemcpyAsync(pn + (size_t)a * np, hn[a], 4 * (size_t)np, cudaMemcpyHostToDevice, c->stream));
    ASOHF_CUDA(cudaMemcpyAsync(pr + (size_t)a * np, hr[a], 4 * (size_t)np, cudaMemcpyHostToDevice, c->stream));
  }
  if (!on_device) {
    ASOHF_CUDA(cudaMemcpyAsync(dcr, cr01, 4 * pc * (size_t)np, cudaMemcpyHostToDevice, c->stream));
    if (conta11) ASOHF_CUDA(cudaMemcpyAsync(dct, conta11, 4 * pc * (size_t)np, cudaMemcpyHostToDevice, c->stream));
  }
  ASOHF_CUDA(cudaMemsetAsync(solap, 0, pc * (size_t)np, c->stream));
  ASOHF_CUDA(cudaMemsetAsync(cnt, 0, 4 * (size_t)np + 4, c->stream));
  const float dxpa = ldexpf(dx, -ir);                       // DX/(2.**IR)
  const float fix = radx1 - dx * 0.5f + 0.5f * dxpa;        // RXFIX
  int kt_ = ktime_begin(c, "veinsgrid_reduced");
  k_veins_box<<<(3 * np + 255) / 256, 256, 0, c->stream>>>(pn, pr, np, dxpa, fix, g1);
  k_veins_neighbours<<<(np + 7) / 8, 256, 0, c->stream>>>(g1, pn, np, cnt, nullptr, nullptr);
  ASOHF_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, off, np + 1, c->stream));
  c->launches += 3;
  std::vector<int32_t> hoff(np + 1);
  ASOHF_CUDA(cudaMemcpyAsync(hoff.data(), off, 4 * (size_t)(np + 1), cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  const int ne = hoff[np];
  int maxnv = 0;
  for (int i = 0; i < np; i++) maxnv = std::max(maxnv, hoff[i + 1] - hoff[i]);
  if (maxnv > max_neighbours) {
    ktime_end(c, kt_);
    return ASOHF_ERR_CAPACITY;  // the reference stops: more neighbours than NPALEV2
  }
  int32_t* nb = nullptr;
  if (ne > 0) {
    // the list lives in the segment buffer (the arena is sized before the count is known)
    ASOHF_CHECK(seg_reserve(c, 4 * (size_t)ne + 256));
    nb = (int32_t*)seg_alloc(c, 4 * (size_t)ne);
    if (!nb) return ASOHF_ERR_CAPACITY;
    k_veins_neighbours<<<(np + 7) / 8, 256, 0, c->stream>>>(g1, pn, np, nullptr, off, nb);
    c->launches++;
  }
  std::vector<int32_t> hnb(ne > 0 ? ne : 1);
  if (ne > 0) ASOHF_CUDA(cudaMemcpyAsync(hnb.data(), nb, 4 * (size_t)ne, cudaMemcpyDeviceToHost, c->stream));
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  // waves: one past the latest wave of the lower-index neighbours
  std::vector<int32_t> wave(np, 0);
  int nwave = 0;
  for (int i = 0; i < np; i++) {
    int w = 0;
    for (int k = hoff[i]; k < hoff[i + 1]; k++)
      if (hnb[k] < i) w = std::max(w, wave[hnb[k]] + 1);
    wave[i] = w;
    nwave = std::max(nwave, w + 1);
  }
  std::vector<int32_t> wstart(nwave + 1, 0), horder(np);
  std::vector<int> wmax(nwave, 0);  // most neighbours of a row of the wave
  for (int i = 0; i < np; i++) {
    wstart[wave[i] + 1]++;
    wmax[wave[i]] = std::max(wmax[wave[i]], hoff[i + 1] - hoff[i]);
  }
  for (int w = 0; w < nwave; w++) wstart[w + 1] += wstart[w];
  {
    std::vector<int32_t> fillp(wstart.begin(), wstart.end() - 1);
    for (int i = 0; i < np; i++) horder[fillp[wave[i]]++] = i;
  }
  ASOHF_CUDA(cudaMemcpyAsync(rows, horder.data(), 4 * (size_t)np, cudaMemcpyHostToDevice, c->stream));
  for (int w = 0; w < nwave; w++) {
    const int nr = wstart[w + 1] - wstart[w];
    if (nr <= 0) continue;
    const dim3 grid((unsigned)nr, (unsigned)std::max(1, std::min(wmax[w], 65535)));
    k_veins_rows<<<grid, 256, 0, c->stream>>>(rows + wstart[w], off, nb, pn, pr, np, dxpa, solap, dcr, dct);
    c->launches++;
  }
  ktime_end(c, kt_);
  ASOHF_CUDA(cudaGetLastError());
  if (!on_device) {
    ASOHF_CUDA(cudaMemcpyAsync(cr01, dcr, 4 * pc * (size_t)np, cudaMemcpyDeviceToHost, c->stream));
    if (conta11) ASOHF_CUDA(cudaMemcpyAsync(conta11, dct, 4 * pc * (size_t)np, cudaMemcpyDeviceToHost, c->stream));
  }
  ASOHF_CUDA(cudaStreamSynchronize(c->stream));
  return ASOHF_OK;
}

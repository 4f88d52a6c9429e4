// Particle text on the device: CSV ingest (read_csv, io.cc:122-178) and the
// VTK snapshot (write_vtk, io.cc:180-195).
//
// Ingest: the text is copied to the device once; line starts come from a
// newline count per 16 KB tile, a scan of the tile counts and an ordered
// emit of the newline positions; then one thread per line parses it as
// io.cc's parse_lines/parse_field do (blanks around fields, ',' between the
// eight fields id,mass,x,y,z,vx,vy,vz, an optional '\r' at the end; a line
// of blanks is skipped; anything else is a malformed line), with the exact
// number conversion of bhg_decimal.cuh; valid lines are compacted in order.
// The header rule of read_csv (skip the first line if its first field is
// not an id) is applied by the host, which sees the first line anyway.
//
// Snapshot: one thread per particle formats its three lines ("x y z",
// "mass", "vx vy vz", numbers as an ostream writes them) in shared memory; the
// block packs its lines and writes them as one piece per section; a scan of
// the pieces' lengths places them in the output.
#include "bhg_kernels.h"
#include "bhg_decimal.cuh"

namespace bhg {

namespace {

constexpr int kTileBytes = 16384;
constexpr int kCsvThreads = 256;  // per block; each thread scans 64 bytes of a tile
static_assert(kTileBytes == kCsvThreads * 64, "tile = threads x 64 bytes");

__device__ __forceinline__ uint32_t count_byte(uint32_t w, uint32_t c4) {
  // bytes of w equal to the byte replicated in c4 (exact, no false positives)
  const uint32_t x = w ^ c4;
  const uint32_t t = ((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x;
  return __popc(~t & 0x80808080u);
}

// newlines in [i0, i1) of the text (byte loop at the ends, words inside)
__device__ uint32_t count_nl(const char* text, size_t i0, size_t i1) {
  uint32_t c = 0;
  size_t i = i0;
  for (; i < i1 && (i & 3); ++i) c += text[i] == '\n';
  for (; i + 4 <= i1; i += 4) c += count_byte(*reinterpret_cast<const uint32_t*>(text + i), 0x0a0a0a0au);
  for (; i < i1; ++i) c += text[i] == '\n';
  return c;
}

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? sh[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane < nw) sh[lane] = s;
  }
  __syncthreads();
  total = sh[(blockDim.x >> 5) - 1];
  const uint32_t base = warp ? sh[warp - 1] : 0u;
  __syncthreads();
  return base + incl - v;
}

}  // namespace

__global__ void __launch_bounds__(kCsvThreads) k_nl_count(const char* __restrict__ text, size_t n,
                                                          uint32_t* __restrict__ tile_count) {
  __shared__ uint32_t sh[32];
  const size_t t0 = (size_t)blockIdx.x * kTileBytes + (size_t)threadIdx.x * 64;
  const uint32_t c = t0 < n ? count_nl(text, t0, t0 + 64 < n ? t0 + 64 : n) : 0u;
  uint32_t total;
  block_excl_scan(c, sh, total);
  if (threadIdx.x == 0) tile_count[blockIdx.x] = total;
}

// Exclusive scan of counts[0 .. m) in place (one block); total to *total.
__global__ void __launch_bounds__(1024) k_scan_counts(uint32_t* __restrict__ counts, uint32_t m,
                                                      uint64_t* __restrict__ total) {
  __shared__ uint32_t sh[32];
  uint64_t carry = 0;
  for (uint32_t base = 0; base < m; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < m ? counts[i] : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_scan(v, sh, tot);
    if (i < m) counts[i] = (uint32_t)(carry + ex);
    carry += tot;
  }
  if (threadIdx.x == 0) *total = carry;
}

// line_start[0] = 0; line_start[k + 1] = 1 + position of newline k.
__global__ void __launch_bounds__(kCsvThreads) k_nl_emit(const char* __restrict__ text, size_t n,
                                                         const uint32_t* __restrict__ tile_off,
                                                         uint64_t* __restrict__ line_start) {
  __shared__ uint32_t sh[32];
  const size_t t0 = (size_t)blockIdx.x * kTileBytes + (size_t)threadIdx.x * 64;
  const size_t t1 = t0 + 64 < n ? t0 + 64 : n;
  const uint32_t c = t0 < n ? count_nl(text, t0, t1) : 0u;
  uint32_t total;
  uint64_t k = (uint64_t)tile_off[blockIdx.x] + block_excl_scan(c, sh, total);
  if (blockIdx.x == 0 && threadIdx.x == 0) line_start[0] = 0;
  for (size_t i = t0; i < t1 && c; ++i)
    if (text[i] == '\n') line_start[1 + k++] = i + 1;
}

namespace {

__device__ __forceinline__ const char* skip_blanks(const char* p, const char* end) {
  while (p < end && (*p == ' ' || *p == '\t')) ++p;
  return p;
}

// parse_field (io.cc:76-91) for the id: std::from_chars into uint32
__device__ bool field_id(const char*& p, const char* end, uint32_t& out) {
  p = skip_blanks(p, end);
  const char* q = p;
  uint64_t v = 0;
  while (q < end && *q >= '0' && *q <= '9') {
    v = v * 10 + (uint64_t)(*q - '0');
    if (v > 0xffffffffull) return false;  // result_out_of_range
    ++q;
  }
  if (q == p) return false;
  out = (uint32_t)v;
  q = skip_blanks(q, end);
  if (q >= end || *q != ',') return false;
  p = q + 1;
  return true;
}

// parse_field for a double (one out-of-line copy: the conversion is large,
// and seven inlined copies would not stay in the instruction cache)
__device__ __noinline__ bool field_f64(const char*& p, const char* end, double& out, bool last, dec::Big& w, dec::Big& b) {
  p = skip_blanks(p, end);
  const char* q;
  if (dec::parse_double(p, end, &out, &q, w, b) != dec::kOk) return false;
  q = skip_blanks(q, end);
  if (last) {
    if (q < end && *q == '\r') ++q;
    if (q != end) return false;
  } else {
    if (q >= end || *q != ',') return false;
    ++q;
  }
  p = q;
  return true;
}

}  // namespace

// One thread per line: lines [first, nlines).  keep[i - first] = 1 for a
// particle line, 0 for a blank one; *bad = the smallest malformed line.
__global__ void __launch_bounds__(128) k_csv_parse(const char* __restrict__ text, size_t n,
                                                   const uint64_t* __restrict__ line_start, uint64_t first,
                                                   uint64_t nlines, Particle* __restrict__ out,
                                                   uint32_t* __restrict__ keep, unsigned long long* __restrict__ bad) {
  dec::Big w, b;
  for (uint64_t i = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nlines;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const char* line = text + line_start[i];
    const char* eol = i + 1 < nlines ? text + line_start[i + 1] - 1 : text + n;
    const char* p = skip_blanks(line, eol);
    uint32_t k = 0;
    if (p != eol && *p != '\r') {
      Particle q;
      q.pad = 0;
      if (field_id(p, eol, q.id) && field_f64(p, eol, q.mass, false, w, b) && field_f64(p, eol, q.pos[0], false, w, b) &&
          field_f64(p, eol, q.pos[1], false, w, b) && field_f64(p, eol, q.pos[2], false, w, b) &&
          field_f64(p, eol, q.vel[0], false, w, b) && field_f64(p, eol, q.vel[1], false, w, b) &&
          field_f64(p, eol, q.vel[2], true, w, b)) {
        out[i - first] = q;
        k = 1;
      } else {
        atomicMin(bad, (unsigned long long)i);
      }
    }
    keep[i - first] = k;
  }
}

// Per-block sums of keep[] (blocks of kCsvThreads entries).
__global__ void __launch_bounds__(kCsvThreads) k_keep_count(const uint32_t* __restrict__ keep, uint64_t m,
                                                            uint32_t* __restrict__ block_count) {
  const uint64_t i = (uint64_t)blockIdx.x * kCsvThreads + threadIdx.x;
  const int c = __syncthreads_count(i < m && keep[i]);
  if (threadIdx.x == 0) block_count[blockIdx.x] = (uint32_t)c;
}

// Kept particles, in order, to dst.
__global__ void __launch_bounds__(kCsvThreads) k_keep_scatter(const Particle* __restrict__ src,
                                                              const uint32_t* __restrict__ keep, uint64_t m,
                                                              const uint32_t* __restrict__ block_off,
                                                              Particle* __restrict__ dst) {
  __shared__ uint32_t sh[32];
  const uint64_t i = (uint64_t)blockIdx.x * kCsvThreads + threadIdx.x;
  const uint32_t k = i < m ? keep[i] : 0u;
  uint32_t total;
  const uint32_t ex = block_excl_scan(k, sh, total);
  if (k) dst[(uint64_t)block_off[blockIdx.x] + ex] = src[i];
}

// ---- snapshot ------------------------------------------------------------------

// The sections of a snapshot: positions, masses, velocities.  A particle's
// line is at most 3 * 13 + 3 bytes ("x y z\n") or 14 ("m\n").  A block formats
// a tile of kVtkTile particles; its text of a section goes, packed, to the
// tile's piece of that section's buffer, and from there to its place.
// Formatting used to write every character to a slot of its own particle in
// device memory, and a gather copied them byte by byte: 226 + 195 us for
// 500,009 particles; now 221 + 62 in four parts, most of it the conversions.
namespace {

constexpr int kVtkTile = 128;
constexpr int kLine[3] = {42, 14, 42};
__device__ constexpr int kLineDev[3] = {42, 14, 42};
static_assert(kVtkTile * 14 % 16 == 0 && kVtkTile * 42 % 16 == 0, "16-byte pieces");

// Inclusive scan of a block of kVtkTile threads, three 21-bit lengths at once.
__device__ __forceinline__ uint64_t block_incl_scan3(uint64_t v, uint64_t* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) sh[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v += sh[w];
  return v;
}

}  // namespace

// Tiles [tile0, tile0 + gridDim.x): text to pieces[k] + tile * kVtkTile *
// kLine[k], lengths to sums[k * tiles + tile].
__global__ void __launch_bounds__(kVtkTile) k_vtk_format(const Particle* __restrict__ p, uint32_t n, uint32_t tile0,
                                                         uint32_t tiles, char* __restrict__ pieces,
                                                         uint32_t* __restrict__ sums) {
  __shared__ char line[kVtkTile * 42];
  __shared__ __align__(16) char text[kVtkTile * 42];
  __shared__ uint64_t sh[kVtkTile / 32];
  dec::Big a, b;
  const uint32_t tile = tile0 + blockIdx.x, i = tile * kVtkTile + threadIdx.x;
  char* piece = pieces;
  for (int k = 0; k < 3; ++k) {
    char* o = line + threadIdx.x * 42;
    int l = 0;
    if (i < n) {
      const double* v = k == 0 ? p[i].pos : k == 1 ? &p[i].mass : p[i].vel;
      const int m = k == 1 ? 1 : 3;
      for (int d = 0; d < m; ++d) {
        l += dec::format_g6(v[d], o + l, a, b);
        o[l++] = d < m - 1 ? ' ' : '\n';
      }
    }
    const uint32_t end = (uint32_t)block_incl_scan3((uint64_t)l, sh);
    char* t = text + (end - (uint32_t)l);
    for (int c = 0; c < l; ++c) t[c] = o[c];
    if (threadIdx.x == kVtkTile - 1) sums[(size_t)k * tiles + tile] = end;
    __syncthreads();
    const uint32_t total = (uint32_t)(sh[0] + sh[1] + sh[2] + sh[3]);
    const int room = kVtkTile * kLineDev[k];
    uint4* dst = reinterpret_cast<uint4*>(piece + (size_t)tile * room);
    for (uint32_t c = threadIdx.x; c < (total + 15) / 16; c += kVtkTile) dst[c] = reinterpret_cast<const uint4*>(text)[c];
    piece += (size_t)tiles * room;
    __syncthreads();
  }
}

// Places of tiles [tile0, tile0 + count) in section blockIdx.x, after what
// totals[] holds of it; the new totals also go to host memory.
__global__ void __launch_bounds__(1024) k_vtk_offsets(const uint32_t* __restrict__ sums, uint32_t tiles, uint32_t tile0,
                                                      uint32_t count, uint64_t* __restrict__ off, uint64_t* totals,
                                                      uint64_t* host_totals) {
  __shared__ uint32_t sh[32];
  const size_t at = (size_t)blockIdx.x * tiles + tile0;
  uint64_t carry = totals[blockIdx.x];
  for (uint32_t base = 0; base < count; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t tot;
    const uint32_t ex = block_excl_scan(i < count ? sums[at + i] : 0u, sh, tot);
    if (i < count) off[at + i] = carry + ex;
    carry += tot;
  }
  __syncthreads();
  if (threadIdx.x == 0) totals[blockIdx.x] = carry, host_totals[blockIdx.x] = carry;
}

// A tile's pieces to their places: words of the destination, each from the two
// source words it straddles, and single bytes at the ends.
__global__ void __launch_bounds__(kVtkTile) k_vtk_place(const char* __restrict__ pieces, const uint32_t* __restrict__ sums,
                                                        uint32_t tiles, uint32_t tile0, const uint64_t* __restrict__ off,
                                                        char* __restrict__ out0, char* __restrict__ out1,
                                                        char* __restrict__ out2) {
  const uint32_t tile = tile0 + blockIdx.x;
  const char* piece = pieces;
  for (int k = 0; k < 3; ++k) {
    const int room = kVtkTile * kLineDev[k];
    const char* src = piece + (size_t)tile * room;
    char* dst = (k == 0 ? out0 : k == 1 ? out1 : out2) + off[(size_t)k * tiles + tile];
    const uint32_t len = sums[(size_t)k * tiles + tile];
    const uint32_t head = min(len, (uint32_t)(-(intptr_t)dst & 3));  // bytes before the first whole word
    const uint32_t words = (len - head) / 4, tail = head + 4 * words;
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(src);
    uint32_t* dw = reinterpret_cast<uint32_t*>(dst + head);
    // the last word's upper source word may lie past the text, not past the piece: head > 0 leaves a byte there
    for (uint32_t w = threadIdx.x; w < words; w += kVtkTile)
      dw[w] = head ? __funnelshift_r(sw[w], sw[w + 1], 8 * head) : sw[w];
    if (threadIdx.x < head) dst[threadIdx.x] = src[threadIdx.x];
    if (threadIdx.x < len - tail) dst[tail + threadIdx.x] = src[tail + threadIdx.x];
    piece += (size_t)tiles * room;
  }
}

// ---- launchers -----------------------------------------------------------------

size_t csv_tiles(size_t nbytes) { return (nbytes + kTileBytes - 1) / kTileBytes; }

void launch_csv_count(const char* text, size_t n, uint32_t* tile_count, uint64_t* total, cudaStream_t s) {
  const size_t tiles = csv_tiles(n);
  if (tiles == 0) return;
  k_nl_count<<<(unsigned)tiles, kCsvThreads, 0, s>>>(text, n, tile_count);
  k_scan_counts<<<1, 1024, 0, s>>>(tile_count, (uint32_t)tiles, total);
}

void launch_csv_emit(const char* text, size_t n, const uint32_t* tile_off, uint64_t* line_start, cudaStream_t s) {
  const size_t tiles = csv_tiles(n);
  if (tiles == 0) return;
  k_nl_emit<<<(unsigned)tiles, kCsvThreads, 0, s>>>(text, n, tile_off, line_start);
}

void launch_csv_parse(const char* text, size_t n, const uint64_t* line_start, uint64_t first, uint64_t nlines,
                      Particle* tmp, uint32_t* keep, unsigned long long* bad, int sms, cudaStream_t s) {
  const uint64_t m = nlines > first ? nlines - first : 0;
  if (m == 0) return;
  uint64_t blocks = (m + 127) / 128;
  if (blocks > (uint64_t)sms * 16) blocks = (uint64_t)sms * 16;
  k_csv_parse<<<(unsigned)blocks, 128, 0, s>>>(text, n, line_start, first, nlines, tmp, keep, bad);
}

size_t csv_keep_blocks(uint64_t m) { return (size_t)((m + kCsvThreads - 1) / kCsvThreads); }

void launch_csv_compact(const Particle* tmp, const uint32_t* keep, uint64_t m, uint32_t* block_count,
                        uint64_t* total, Particle* dst, cudaStream_t s) {
  const size_t blocks = csv_keep_blocks(m);
  if (blocks == 0) return;
  k_keep_count<<<(unsigned)blocks, kCsvThreads, 0, s>>>(keep, m, block_count);
  k_scan_counts<<<1, 1024, 0, s>>>(block_count, (uint32_t)blocks, total);
  if (dst) k_keep_scatter<<<(unsigned)blocks, kCsvThreads, 0, s>>>(tmp, keep, m, block_count, dst);
}

uint32_t vtk_tiles(uint32_t n) { return (uint32_t)(((uint64_t)n + kVtkTile - 1) / kVtkTile); }
size_t vtk_section_bytes(uint32_t n, int k) { return (size_t)vtk_tiles(n) * kVtkTile * kLine[k]; }
size_t vtk_piece_bytes(uint32_t n) {
  return vtk_section_bytes(n, 0) + vtk_section_bytes(n, 1) + vtk_section_bytes(n, 2);
}

size_t vtk_most_bytes(uint32_t n) { return (size_t)n * (kLine[0] + kLine[1] + kLine[2]); }

void launch_vtk_tiles(const Particle* p, uint32_t n, uint32_t tile0, uint32_t count, char* pieces, uint32_t* sums,
                      uint64_t* off, uint64_t* totals, uint64_t* host_totals, char* const out[3], cudaStream_t s) {
  if (count == 0) return;
  const uint32_t tiles = vtk_tiles(n);
  k_vtk_format<<<count, kVtkTile, 0, s>>>(p, n, tile0, tiles, pieces, sums);
  k_vtk_offsets<<<3, 1024, 0, s>>>(sums, tiles, tile0, count, off, totals, host_totals);
  k_vtk_place<<<count, kVtkTile, 0, s>>>(pieces, sums, tiles, tile0, off, out[0], out[1], out[2]);
}

}  // namespace bhg

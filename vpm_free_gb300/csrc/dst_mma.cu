// dst_mma.cu -- DST-I lines as matrix products on the tensor cores.
//
// X_k = sum_j x_j sin(pi j k / N), k = 1..n, N = n + 1.  With the line folded,
// P_j = x_j + x_{N-j} and M_j = x_j - x_{N-j} (j <= N/2, the middle one alone),
// odd k need P and even k need M: two products with half-size sine matrices.
// An FFT costs about 25 FP64 operations per value on a pipe of two lanes per
// clock and SM, which held the passes at 0.16 to 0.2 ms per 10^7 values; as a
// product a value needs none.  The line becomes 55-bit integers at the scale
// of its own largest magnitude, the folds are integer sums (no rounding), and
// seven balanced base-256 digits of them and of the matrix, held as FP16, meet
// in the 28 of 49 digit products with i + j <= 6, accumulated in FP32 by i + j.
// The six sums up to i + j = 5 are exact: with every digit of the line at its
// largest (128, the top one 256) and the digits of the sine matrices as they
// are, for all N up to 417 and factors in [1, 2), they stay below 0.91 2^24.
// The seventh can reach 1.01 2^24; its rounding is below the nine bits that the
// joined integer drops.  That integer is rounded once to double.  The error is
// that of rounding the line's values and the sines to 55 bits and of the dropped
// products, of which the six with i + j = 7 reach 2^-53.4 of a product's scale at
// worst; as digits of either sign they are a seventh of that (root mean square)
// and add up as the root of K.
//
// Tile: 64 lines (columns) x 128 outputs of one parity (rows), seven
// accumulators of 64 columns in tensor memory; the lines' digits stay in
// shared memory (910 bytes per folded index), the matrix streams through a
// ring of 16-k pieces, loaded by one warp while another issues the products.
// K is dealt over the digit array as k = 1 + g + G m (m = 0..7 within a
// 16-byte piece, G pieces), so that consecutive threads read consecutive
// values along x.  The line's scale needs a first reading of its values; the
// next tile's runs beside this tile's last product.  Per tile at N = 256
// (94 thousand clocks): 36 the products (57 clocks each, shared-memory reads
// of the operands; issue and matrix pieces the rest), 23 the digits, 22 the
// outputs, 13 the scale before it moved beside the product.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "dst_mma.h"
#include "tc05.cuh"

namespace vpmg {

namespace {

constexpr int kLines = 64;
constexpr int kThreads = 512;
constexpr int kRows = 128;
constexpr int kDigits = 7;
constexpr int kPiece = 2 * kRows * 16;          // one digit, 16 k, 128 outputs
constexpr int kCol = kLines * 16 + 16;          // 8 k of the lines, padded against bank conflicts
constexpr int kSmemMax = 227 * 1024 - 3584;  // 3.3 KB are static
constexpr int kMaxSlots = 6;
// The ring's pieces: 16 k of all seven digits (28 KB, one bulk copy) where two
// fit, else of digits 0..2 and 3..6 in turn (bulk copies of 4 KB, one digit
// each, held the products to 147 clocks each instead of 60).
constexpr int kSlot[3] = {0, 7 * kPiece, 4 * kPiece};

__host__ __device__ __forceinline__ int dst_kp(int n) { return (((n + 1) / 2) + 15) & ~15; }  // padded folded length
__host__ __device__ __forceinline__ int dst_count(int n, int par) { return par ? n / 2 : (n + 1) / 2; }
__host__ __device__ __forceinline__ int dst_mtiles(int n, int par) { return (dst_count(n, par) + kRows - 1) / kRows; }

// Piece (par, mt, ks, digit) of the matrix times factor in [1, 2): rows m,
// k positions 16 ks + 8 g' + i <-> j = 1 + g + G i with g = 2 ks + g'.
struct DstTables {
  DstTable t[3];
  int block0[4];  // first block of each
};
__global__ void k_dst_table(const DstTables A) {
  const int bx = (int)blockIdx.x, job = bx >= A.block0[2] ? 2 : bx >= A.block0[1] ? 1 : 0;
  unsigned char* const T = A.t[job].T;
  const int n = A.t[job].n;
  const double factor = A.t[job].factor;
  const int N = n + 1, kp = dst_kp(n), G = kp / 8, nks = kp / 16;
  const int mt0 = dst_mtiles(n, 0), mts = mt0 + dst_mtiles(n, 1);
  const int t = (bx - A.block0[job]) * (int)blockDim.x + threadIdx.x;  // (mt, ks, g', m)
  if (t >= mts * nks * 2 * kRows) return;
  const int m = t % kRows, gg = (t / kRows) & 1, ks = (t / (2 * kRows)) % nks, mt = t / (2 * kRows * nks);
  const int par = mt >= mt0 ? 1 : 0;
  const int o = (par ? mt - mt0 : mt) * kRows + m;
  const int k = 2 * o + 1 + par;
  unsigned d[4][kDigits];
  long long x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int j = 1 + (2 * ks + gg) + G * i;
    double s = 0.0;
    if (k <= n && j <= N / 2) s = sinpi((double)((unsigned)j * k % (2u * N)) / N) * factor;
    x[i] = (long long)rint(s * 36028797018963968.0);  // 2^55
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) tc05::digits256x2(x[2 * i], x[2 * i + 1], d[i]);
#pragma unroll
  for (int j = 0; j < kDigits; ++j)
    reinterpret_cast<uint4*>(T + ((size_t)(mt * nks + ks) * kDigits + j) * kPiece)[gg * kRows + m] =
        make_uint4(d[0][j], d[1][j], d[2][j], d[3][j]);
}

struct DstArgs {
  const unsigned char* T;
  const double* in;
  const double* sol;   // x forward: boundary values
  double* out;
  int n, nlines, ntile, nc, slots, np;  // np: pieces per 16 k
  int shift, neg;      // outputs times 2^shift, negated
  int zero_bc;
  int m0, m1, m2;
  long long sy, sz, o;  // node strides and the offset of the first interior node (x passes)
  size_t ics, scs, ocs;
  double ihx2, ihy2, ihz2;
  int polls;     // limit of every wait
  int* status;   // null or the word that gets kErrWait when a wait runs out
};

// V 2^e as a double, rounded to nearest even.
__device__ __forceinline__ double to_double(long long V, int e) {
  const unsigned long long sg = (unsigned long long)V & 0x8000000000000000ull;
  unsigned long long W = (unsigned long long)(V < 0 ? -V : V);
  if (W == 0) return 0.0;
  const int lz = __clzll((long long)W);
  W <<= lz;
  const int be = 63 - lz + e + 1023;  // biased exponent before rounding
  if (be < 1 || be > 2045) {
    const double v = scalbn((double)W, e - lz);
    return sg ? -v : v;
  }
  const unsigned long long r = W + 0x3FFull + ((W >> 11) & 1ull);
  // a carry out of the 64 bits is the next power of two
  const unsigned long long mant = r < W ? 0x20000000000000ull : r >> 11;
  return __longlong_as_double((long long)((((unsigned long long)(be - 1) << 52) + mant) | sg));
}

// MODE 0: x forward (node array -> lines), 1: y, 2: x inverse (lines -> node array)
//
// Every wait has a limit.  When one runs out, the thread that waited stops
// loading or issuing; the barrier behind each product tells the whole CTA, which
// waits for its own copies and products in flight, sets *status, writes NaN to
// the outputs of this tile and of those it still had, and ends.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1) k_dst_mma(const __grid_constant__ DstArgs P) {
  extern __shared__ __align__(128) unsigned char dst_sm[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxSlots + 2];
  __shared__ uint32_t tslot;
  // the lines of this tile and of the next (its magnitudes are taken while this one's last product runs)
  __shared__ long long loff[2][kLines], ooff[2][kLines];  // first value of each line, read and written
  __shared__ int lflag[2][kLines];     // bit 0: line exists; 1..4: next to the box's y and z faces
  __shared__ unsigned emax[2][kLines];
  __shared__ int some[2];              // any value not zero
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = P.n, N = n + 1, J = N / 2, kp = dst_kp(n), G = kp / 8, nks = kp / 16;
  const uint32_t dig = tc05::smem_u32(dst_sm);
  const uint32_t ring = dig + (uint32_t)(kDigits * G * kCol);
  unsigned char* const stage = dst_sm + (size_t)kDigits * G * kCol;
  const uint32_t full = tc05::smem_u32(bars), empty = full + 8 * kMaxSlots, done = full + 16 * kMaxSlots;
  const uint32_t drained = done + 8;
  if (warp == 0) tc05::tmem_alloc(tc05::smem_u32(&tslot), 512);
  if (tid == 0) {
    for (int i = 0; i < 2 * kMaxSlots + 2; ++i) tc05::bar_init(full + 8 * i, 1);
    tc05::bar_init_fence();
  }
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tb = tslot;
  constexpr uint32_t idesc = tc05::idesc_f16(kRows, kLines);
  bool dead = false, failed = false;
  const int S = P.slots, np = P.np;
  const uint32_t sbytes = np == 1 ? 7 * kPiece : 4 * kPiece;
  // the loading thread's (warp 1) and the issuing thread's (warp 0) place in the ring
  int slot = 0;
  uint32_t phase = 0, wrapped = 0, ndone = 0;
  uint32_t loads = 0;  // pieces loaded by this thread
  const long long estr = MODE == 1 ? P.m0 : 1;  // doubles between a line's values
  const int ntot = P.ntile * P.nc;
  auto in_of = [&](int tile) { return P.in + (size_t)(tile / P.ntile) * P.ics; };
  auto sol_of = [&](int tile) { return MODE == 0 ? P.sol + (size_t)(tile / P.ntile) * P.scs : nullptr; };
  auto lines_of = [&](int tile, int q) {  // tid < kLines
    const int l = (tile % P.ntile) * kLines + tid;
    long long off = 0, oo = 0;
    int fl = 0;
    if (l < P.nlines) {
      fl = 1;
      if (MODE == 0) {
        const int c = l / P.m1, j = l - c * P.m1;
        off = P.o + P.sy * j + P.sz * c;
        oo = (long long)l * n;
        fl |= (j == 0 ? 2 : 0) | (j == P.m1 - 1 ? 4 : 0) | (c == 0 ? 8 : 0) | (c == P.m2 - 1 ? 16 : 0);
      } else if (MODE == 1) {
        off = oo = (long long)(l % P.m0) + (long long)P.m0 * P.m1 * (l / P.m0);
      } else {
        off = (long long)l * n;
        oo = P.o + P.sy * (l % P.m1) + P.sz * (l / P.m1);
      }
    }
    loff[q][tid] = off;
    ooff[q][tid] = oo;
    lflag[q][tid] = fl;
    emax[q][tid] = 0;
    if (tid == 0) some[q] = 0;
  };
  // x forward: the boundary values that fold into value v = line[j] at `at`.
  // Few values have any; callers load plainly and correct those (tests beside
  // every load held the pass with given faces to twice the other passes' time).
  auto ends = [&](const double* sol, double v, long long at, int j) {
    if (j == 1) v -= sol[at - 1] * P.ihx2;
    if (j == n) v -= sol[at + 1] * P.ihx2;
    return v;
  };
  // nodes beyond the y and z faces next to a line: offset and factor of flag bit 1 + f
  auto side = [&](int f, double& h) -> long long {
    h = f < 2 ? P.ihy2 : P.ihz2;
    return f == 0 ? -P.sy : f == 1 ? P.sy : f == 2 ? -P.sz : P.sz;
  };
  const bool faces = MODE == 0 && !P.zero_bc;
  // the largest magnitude of each line of `tile`, by the warps from w0 on
  auto magnitudes = [&](int tile, int q, int w0) {
    const double* in = in_of(tile);
    const double* sol = sol_of(tile);
    unsigned any = 0;
    constexpr int U = 8;  // loads in flight
    if (MODE == 1) {
      const int line = tid & (kLines - 1), fl = lflag[q][line];
      const int step = (kThreads - 32 * w0) / kLines;
      const long long at = loff[q][line];
      unsigned m = 0;
      if (fl & 1)
        for (int j0 = 1 + (tid - 32 * w0) / kLines; j0 <= n; j0 += U * step) {
          double v[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            v[u] = j0 + u * step <= n ? in[at + estr * (j0 + u * step - 1)] : 0.0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            m = max(m, (unsigned)__double2hiint(v[u]) & 0x7FFFFFFFu);
            any |= v[u] != 0.0;
          }
        }
      if (m) atomicMax(&emax[q][line], m);
    } else {
      for (int line = warp - w0; line < kLines; line += kThreads / 32 - w0) {
        const int fl = lflag[q][line];
        const long long at = loff[q][line];
        unsigned m = 0;
        if (fl & 1)
          for (int j0 = 1 + lane; j0 <= n; j0 += U * 32) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              v[u] = j0 + u * 32 <= n ? in[at + j0 + u * 32 - 1] : 0.0;
            if (faces) {
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int j = j0 + u * 32;
                if (j == 1 || j == n) v[u] = ends(sol, v[u], at + j - 1, j);
              }
              for (int f = 0; f < 4; ++f)
                if (fl >> (f + 1) & 1) {
                  double h, q[U];
                  const double* const p = sol + at + side(f, h) - 1;
#pragma unroll
                  for (int u = 0; u < U; ++u) q[u] = j0 + u * 32 <= n ? p[j0 + u * 32] : 0.0;
#pragma unroll
                  for (int u = 0; u < U; ++u) v[u] -= q[u] * h;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              m = max(m, (unsigned)__double2hiint(v[u]) & 0x7FFFFFFFu);
              any |= v[u] != 0.0;
            }
          }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) emax[q][line] = m;
      }
    }
    if (any) some[q] = 1;
  };
  int tile = blockIdx.x, cur = 0;
  if (tile < ntot && tid < kLines) lines_of(tile, 0);
  __syncthreads();
  if (tile < ntot) magnitudes(tile, 0, 0);
  for (; tile < ntot && !failed; tile += gridDim.x, cur ^= 1) {
    __syncthreads();
    const int next = tile + gridDim.x;
    if (next < ntot && tid < kLines) lines_of(next, cur ^ 1);
    const double* in = in_of(tile);
    const double* sol = sol_of(tile);
    double* out = P.out + (size_t)(tile / P.ntile) * P.ocs;
    if (!some[cur]) {
      // zero lines transform to zero
      for (int t = tid; t < kLines * n; t += kThreads) {
        const int line = MODE == 1 ? t & (kLines - 1) : t / n, k = MODE == 1 ? t / kLines : t - line * n;
        if (lflag[cur][line] & 1) out[ooff[cur][line] + estr * k] = 0.0;
      }
      __syncthreads();
      if (next < ntot) magnitudes(next, cur ^ 1, 0);
      continue;
    }
    // digits of 8 folded values: unit u = (line, piece g)
    auto digits = [&](int u, int par, unsigned d[4][kDigits]) {
      const int line = MODE == 1 ? u & (kLines - 1) : u / G;
      const int g = MODE == 1 ? u / kLines : u - line * G;
      const int fl = lflag[cur][line];
      const long long at = loff[cur][line] - estr;
      const int E = tc05::scale_exp(emax[cur][line]);
      double a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int j = 1 + g + G * i;
        a[i] = (fl & 1) && j <= J ? in[at + estr * j] : 0.0;
        b[i] = (fl & 1) && j <= J && N - j != j ? in[at + estr * (N - j)] : 0.0;
      }
      if (faces && (fl & 1)) {
        if (g == 0) {  // j = 1 and n
          a[0] = ends(sol, a[0], at + 1, 1);
          if (n > 1) b[0] = ends(sol, b[0], at + n, n);
        }
        for (int f = 0; f < 4; ++f)
          if (fl >> (f + 1) & 1) {
            double h, qa[8], qb[8];
            const double* const p = sol + at + side(f, h);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int j = 1 + g + G * i;
              qa[i] = j <= J ? p[j] : 0.0;
              qb[i] = j <= J && N - j != j ? p[N - j] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              a[i] -= qa[i] * h;
              b[i] -= qb[i] * h;
            }
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        long long x[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const long long p = tc05::fixed55(a[2 * i + h], E), q = tc05::fixed55(b[2 * i + h], E);
          x[h] = par ? p - q : p + q;
        }
        tc05::digits256x2(x[0], x[1], d[i]);
      }
    };
    auto store = [&](int u, const unsigned d[4][kDigits]) {
      const int line = MODE == 1 ? u & (kLines - 1) : u / G;
      const int g = MODE == 1 ? u / kLines : u - line * G;
#pragma unroll
      for (int j = 0; j < kDigits; ++j)
        *reinterpret_cast<uint4*>(dst_sm + (size_t)(j * G + g) * kCol + line * 16) =
            make_uint4(d[0][j], d[1][j], d[2][j], d[3][j]);
    };
    const int units = kLines * G;
    int mt = 0;
    for (int par = 0; par < 2 && !failed; ++par) {
      const int cnt = dst_count(n, par), mts = dst_mtiles(n, par);
      for (int u = tid; u < units; u += kThreads) {
        unsigned d[4][kDigits];
        digits(u, par, d);
        store(u, d);
      }
      tc05::fence_async();
      __syncthreads();
      for (int h = 0; h < mts; ++h, ++mt) {
        if (warp == 1) {  // the matrix, piece by piece
          if (lane == 0) {
            const unsigned char* src = P.T + (size_t)mt * nks * kDigits * kPiece;
            for (int i = 0; i < nks * np; ++i) {
              const uint32_t bytes = np == 1 ? 7 * kPiece : (i & 1) ? 4 * kPiece : 3 * kPiece;
              if (wrapped) tc05::bar_wait(empty + 8 * slot, phase ^ 1u, dead, P.polls);
              if (dead) break;
              ++loads;
              tc05::bar_expect(full + 8 * slot, bytes);
              tc05::bulk_load(ring + slot * sbytes, src, bytes, full + 8 * slot);
              src += bytes;
              if (++slot == S) {
                slot = 0;
                phase ^= 1u;
                wrapped = 1;
              }
            }
          }
          __syncwarp();
        } else if (warp == 0) {  // the products
          if (lane == 0) {
            tc05::fence_after();
            for (int ks = 0; ks < nks && !dead; ++ks) {
              const uint64_t db = tc05::desc(dig + (uint32_t)(2 * ks) * kCol, kCol);
              const uint64_t dj = (uint64_t)((uint32_t)(G * kCol) >> 4);
              uint64_t da = 0;
#pragma unroll
              for (int w = 0; w < kDigits; ++w) {
                if (w == 0 || (w == 3 && np == 2)) {  // the next piece
                  tc05::bar_wait(full + 8 * slot, phase, dead, P.polls);
                  if (dead) break;
                  da = tc05::desc(ring + slot * sbytes, kRows * 16);
                }
#pragma unroll
                for (int j = 0; j < kDigits - w; ++j)
                  tc05::mma(tb + (w + j) * kLines, da, db + j * dj, idesc, (w > 0 || ks > 0) ? 1u : 0u);
                da += kPiece >> 4;
                if (w == kDigits - 1 || (w == 2 && np == 2)) {
                  tc05::commit(empty + 8 * slot);
                  if (++slot == S) {
                    slot = 0;
                    phase ^= 1u;
                  }
                }
              }
            }
            tc05::commit(done);
          }
          __syncwarp();  // the warp's other lanes do not spin beside the issuing one
        } else if (par == 1 && h == mts - 1 && next < ntot) {  // meanwhile: the next tile's magnitudes
          magnitudes(next, cur ^ 1, 2);
        }
        tc05::bar_wait(done, ndone & 1, dead, P.polls);
        ++ndone;
        if (__syncthreads_or(dead)) {
          failed = true;
          break;
        }
        tc05::fence_after();
        // outputs: row m of the tile in lane m, 16 lines per warp
        const int m = 32 * (warp & 3) + lane, cb = 16 * (warp >> 2);
        const int o = h * kRows + m, k = 2 * o + 1 + par;
        const bool any = h * kRows + 32 * (warp & 3) < cnt;
        const uint32_t ta = tb + ((uint32_t)(32 * (warp & 3)) << 16) + cb;
        double* const st = reinterpret_cast<double*>(stage + (size_t)warp * 2048);  // [m][8], columns xor m
#pragma unroll
        for (int c8 = 0; c8 < 2; ++c8) {
          if (!any) break;  // rows past the last output (whole warp)
          uint32_t v[kDigits][8];
#pragma unroll
          for (int d = 0; d < kDigits; ++d) tc05::ld8(ta + d * kLines + 8 * c8, v[d]);
          tc05::ld_wait();
          if (MODE == 1) __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int line = cb + 8 * c8 + i;
            auto q = [&](int d) { return (long long)__float2int_rn(__uint_as_float(v[d][i])); };
            // integers: values 2^(1077 - E), sines 2^55, the sums in units of
            // 2^48; |sum| < 208 2^56 2^56 / 2^48, so it fits with 9 bits dropped
            const long long hi = (q(0) << 32) + (q(1) << 24) + (q(2) << 16) + (q(3) << 8) + q(4);
            const long long lo = (q(5) << 8) + q(6);
            const long long V = (hi << 7) + ((lo + 256) >> 9);
            const int E = tc05::scale_exp(emax[cur][line]);
            double r = to_double(P.neg ? -V : V, 57 + E - 1077 - 55 + P.shift);
            if (E >= 0x7FF) r = __longlong_as_double(0x7FF8000000000000ll);
            if (MODE == 1) {
              st[lane * 8 + (i ^ (lane & 7))] = r;
            } else if (o < cnt && (lflag[cur][line] & 1)) {
              out[ooff[cur][line] + (k - 1)] = r;
            }
          }
          if (MODE == 1) {
            __syncwarp();
            // four outputs x eight consecutive lines per store
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              const int mm = 4 * t + (lane >> 3), i = lane & 7, line = cb + 8 * c8 + i;
              const int oo = h * kRows + 32 * (warp & 3) + mm;
              const double r = st[mm * 8 + (i ^ (mm & 7))];
              if (oo < cnt && (lflag[cur][line] & 1)) out[ooff[cur][line] + estr * (2 * oo + par)] = r;
            }
          }
        }
        tc05::fence_before();
        tc05::fence_async();  // digits for the products, and the ring for the bulk copies
        __syncthreads();
      }
    }
  }
  __syncthreads();
  if (failed) {
    bool late = false;  // these waits have the full limit
    if (warp == 0 && lane == 0) {
      tc05::commit(drained);
      tc05::bar_wait(drained, 0, late, tc05::kPolls);
    }
    if (warp == 1 && lane == 0)
      for (uint32_t i = 0; i < (uint32_t)S && i < loads; ++i)  // the last copy into each slot
        tc05::bar_wait(full + 8 * i, ((loads - i - 1) / S) & 1, late, tc05::kPolls);
    __syncwarp();
    if (tid == 0 && P.status) atomicMax(P.status, kErrWait);
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    for (tile -= gridDim.x; tile < ntot; tile += gridDim.x) {  // from the tile that failed
      __syncthreads();
      if (tid < kLines) lines_of(tile, 0);
      __syncthreads();
      double* out = P.out + (size_t)(tile / P.ntile) * P.ocs;
      for (int t = tid; t < kLines * n; t += kThreads) {
        const int line = MODE == 1 ? t & (kLines - 1) : t / n, k = MODE == 1 ? t / kLines : t - line * n;
        if (lflag[0][line] & 1) out[ooff[0][line] + estr * k] = nan;
      }
    }
    __syncthreads();
  }
  if (warp == 0) tc05::tmem_free(tb, 512);
}

// Shared memory left for the ring; pieces per 16 k (0: the lines are too long).
int ring_bytes(int n) { return kSmemMax - kDigits * (dst_kp(n) / 8) * kCol; }
int pieces_for(int n) { return ring_bytes(n) >= 2 * kSlot[1] ? 1 : ring_bytes(n) >= 2 * kSlot[2] ? 2 : 0; }

constexpr int kMaxDev = 64;
bool g_attr[kMaxDev] = {false};
int g_sms[kMaxDev] = {0};
int current_device() {
  int dev = 0;
  VPMG_CUDA(cudaGetDevice(&dev));
  VPMG_CHECK(dev >= 0 && dev < kMaxDev, VPMG_ERR_UNSUPPORTED, "device index beyond the per-device tables");
  return dev;
}
// One CTA fills an SM and the tiles are dealt by a fixed stride: more CTAs than
// SMs would run after the others' whole share.
int sm_count() {
  int& n = g_sms[current_device()];
  if (!n) VPMG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, current_device()));
  return n;
}
template <int MODE>
void launch(DstArgs& A, cudaStream_t s) {
  A.ntile = (A.nlines + kLines - 1) / kLines;
  A.np = pieces_for(A.n);
  VPMG_CHECK(A.np, VPMG_ERR_STATE, "line too long for the product form");
  A.slots = std::min(kMaxSlots, ring_bytes(A.n) / kSlot[A.np]);
  const size_t sm = (size_t)kDigits * (dst_kp(A.n) / 8) * kCol + (size_t)A.slots * kSlot[A.np];
  const int tiles = A.ntile * A.nc;
  if (tiles <= 0) return;
  k_dst_mma<MODE><<<std::min(tiles, sm_count()), kThreads, sm, s>>>(A);
  VPMG_LAUNCHED();
  VPMG_CUDA(cudaGetLastError());
}

}  // namespace

// Lines of N = n + 1 >= 100 intervals whose digits leave room for the ring
// (N <= 416), where the tiles of 64 lines fill the SMs: a tile takes as long
// alone as among one per SM, the FFT's time grows with the lines.  Measured on
// the two x passes of a dense one-component solve, FFT over products, at 35, 66,
// 79, 108, 142, 195 and 302 tiles on 152 SMs:
//   N = 100  0.88 0.95 1.04 1.10 1.16 1.13 1.24    N = 135  0.86 1.09 1.24 1.36 1.49 1.46 1.59
//   N = 160  0.78 0.99 1.10 1.19 1.30 1.18 1.35    N = 165  0.90 1.27 1.32 1.50 1.67 1.51 1.70
//   N = 256  0.80 1.06 1.11 1.19 1.28 1.15 1.29    N = 320  0.65 0.92 0.97 1.10 1.20 1.04 1.23
// (odd N go by FFTs of twice the length).  Hence from 0.55 tiles per SM and
// round, odd N from 0.35.  Tables made for one call weigh as 26 tiles: the
// allocation-free solve of N = 129 takes 0.185 ms with products and 0.132 with
// FFTs at 36 tiles, 0.202 and 0.167 at 63, 0.291 and 0.315 at 143.  Lines of 64
// to 96 intervals gain nothing (a 64^3 step, N = 64 and 80, 1.91 ms by FFT and
// 1.96 by products).  Where most lines are zero, as the right-hand sides of few
// particles in long boxes, the FFT skips more of them: steps on 256 x 48 x 48 and
// 400 x 48 x 48 cells lose 3 and 5 %.
bool dst_mma_wanted(int n, long long lines, int nc, bool once) {
  if (n + 1 < 100 || !pieces_for(n)) return false;
  const double sms = sm_count();
  const double tiles = (double)((lines + kLines - 1) / kLines * nc);
  const double fill = (tiles - (once ? 26.0 : 0.0)) / (std::ceil(tiles / sms) * sms);
  return fill >= ((n + 1) & 1 ? 0.35 : 0.55);
}

int wait_polls() {
  const char* e = std::getenv("VPMG_WAIT_POLLS");
  return e ? std::max(0, std::atoi(e)) : tc05::kPolls;
}

size_t dst_mma_table_bytes(int n) {
  return (size_t)(dst_mtiles(n, 0) + dst_mtiles(n, 1)) * (dst_kp(n) / 16) * kDigits * kPiece;
}

void dst_mma_setup() {
  const int dev = current_device();
  if (!g_attr[dev]) {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    VPMG_CUDA(cudaFuncSetAttribute(k_dst_mma<0>, a, kSmemMax));
    VPMG_CUDA(cudaFuncSetAttribute(k_dst_mma<1>, a, kSmemMax));
    VPMG_CUDA(cudaFuncSetAttribute(k_dst_mma<2>, a, kSmemMax));
    g_attr[dev] = true;
  }
}

void dst_mma_tables(const DstTable* t, int count, cudaStream_t s) {
  VPMG_CHECK(count >= 1 && count <= 3, VPMG_ERR_ARG, "dst_mma_tables: 1..3 tables");
  DstTables A{};
  int blocks = 0;
  for (int i = 0; i < 3; ++i) {
    A.block0[i] = blocks;
    if (i >= count) continue;
    A.t[i] = t[i];
    const int n = t[i].n;
    blocks += ((dst_mtiles(n, 0) + dst_mtiles(n, 1)) * (dst_kp(n) / 16) * 2 * kRows + 127) / 128;
  }
  A.block0[3] = blocks;
  for (int i = count; i < 3; ++i) A.block0[i] = blocks;
  k_dst_table<<<blocks, 128, 0, s>>>(A);
  VPMG_LAUNCHED();
  VPMG_CUDA(cudaGetLastError());
}

static void box_args(DstArgs& A, const DstBox& b) {
  A.n = b.m[0];
  A.nlines = b.m[1] * b.m[2];
  A.m0 = b.m[0]; A.m1 = b.m[1]; A.m2 = b.m[2];
  A.sy = b.dims[0];
  A.sz = (long long)b.dims[0] * b.dims[1];
  A.o = b.o[0] + A.sy * b.o[1] + A.sz * b.o[2];
}

void dst_mma_x_fwd(const unsigned char* T, int shift, int neg, const double* rhs, const double* sol, bool zero_bc,
                   double* out, const DstBox& b, double ihx2, double ihy2, double ihz2, int nc, size_t rcs, size_t scs,
                   size_t ocs, const DstWait& w, cudaStream_t s) {
  DstArgs A{};
  A.polls = w.polls; A.status = w.status;
  box_args(A, b);
  A.T = T;
  A.in = rhs; A.sol = sol; A.out = out;
  A.zero_bc = zero_bc ? 1 : 0;
  A.nc = nc;
  A.shift = shift; A.neg = neg;
  A.ics = rcs; A.scs = scs; A.ocs = ocs;
  A.ihx2 = ihx2; A.ihy2 = ihy2; A.ihz2 = ihz2;
  launch<0>(A, s);
}

void dst_mma_y(const unsigned char* T, const double* in, double* out, int m0, int m1, int m2, int nc, size_t cs,
               const DstWait& w, cudaStream_t s) {
  DstArgs A{};
  A.polls = w.polls; A.status = w.status;
  A.T = T;
  A.n = m1;
  A.nlines = m0 * m2;
  A.m0 = m0; A.m1 = m1; A.m2 = m2;
  A.in = in; A.out = out;
  A.nc = nc;
  A.ics = A.ocs = cs;
  launch<1>(A, s);
}

void dst_mma_x_inv(const unsigned char* T, const double* in, double* sol, const DstBox& b, int nc, size_t ics,
                   size_t scs, const DstWait& w, cudaStream_t s) {
  DstArgs A{};
  A.polls = w.polls; A.status = w.status;
  box_args(A, b);
  A.T = T;
  A.in = in; A.out = sol;
  A.nc = nc;
  A.ics = ics; A.ocs = scs;
  launch<2>(A, s);
}

}  // namespace vpmg

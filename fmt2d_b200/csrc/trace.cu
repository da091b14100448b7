// Host side of the ray backtrace and Frechet rows: device tables of the
// model, the trace (its entries go into a pool of chunks; a second trace where
// the pool was too small) and the assembly of the entries into CSR rows
// (read_frechet_data2d's layout: one row per pick, columns ascending, entries
// with |value| <= 1e-30 dropped as compute_frechet_for_ray2d does,
// src/inversion2d.f90:4761-4768).
#include "engine.h"
#include "rays.cuh"
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>
#include <algorithm>
#include <cmath>

namespace fmt2d {

#define TCK(x)                                                                \
  do {                                                                        \
    cudaError_t e_ = (x);                                                     \
    if (e_ != cudaSuccess) return std::string(#x ": ") + cudaGetErrorString(e_); \
  } while (0)

namespace {

__global__ void k_keep(const double* vals, int n, int* flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  flag[i] = i < n && fabs(vals[i]) > 1.0e-30 ? 1 : 0;
}

// Row starts: the kept entries before a pick's first key (counting them per
// pick with atomics took 2.8 ms for 22 million entries of 30276 picks).
__global__ void k_row_starts(const unsigned long long* keys, const int* pos, int n, int npick,
                             int* row_ptr) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > npick) return;
  const unsigned long long key = (unsigned long long)p << 32;
  int a = 0, b = n;
  while (a < b) {
    const int m = a + (b - a) / 2;
    if (keys[m] < key) a = m + 1;
    else b = m;
  }
  row_ptr[p] = pos[a];
}

__global__ void k_scatter_rows(const unsigned long long* keys, const double* vals,
                               const int* flag, const int* pos, int n, int* col, double* val) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  col[pos[i]] = (int)(keys[i] & 0xffffffffull);
  val[pos[i]] = vals[i];
}

template <class T>
std::string put_vec(DevBuf& b, const T* v, size_t n, cudaStream_t st) {
  b.alloc(std::max<size_t>(n, 1) * sizeof(T));
  if (!b.p) return "device allocation failed";
  if (n) TCK(cudaMemcpyAsync(b.p, v, n * sizeof(T), cudaMemcpyHostToDevice, st));
  return std::string();
}

}  // namespace

std::string Engine::upload_trace_tables() {
  const Model& m = m_;
  std::string e;
  if (!(e = put_vec(d_pvel_, m.vel.data(), m.vel.size(), stream_)).empty()) return e;
  if (!(e = put_vec(d_invidx_, m.inv_idx.data(), m.inv_idx.size(), stream_)).empty()) return e;
  if (!(e = put_vec(d_xpos_, m.xpos.data(), m.xpos.size(), stream_)).empty()) return e;
  TrModel t;
  t.nx = m.nx;
  t.nz = m.nz;
  t.x0 = m.x0;
  t.dx = m.dx;
  t.tol = m.tolerance;
  t.vwater = m.vwater;
  t.xp0 = m.xpos[0];
  t.vdx = m.xpos[1] - m.xpos[0];
  t.rdx = 1.0 / t.dx;
  t.rvdx = 1.0 / t.vdx;
  t.rvwater = 1.0 / t.vwater;
  t.vel = d_pvel_.as<double>();
  t.xpos = d_xpos_.as<double>();
  for (int k = 1; k <= 5; ++k) t.ifz[k] = ifc_buf_[k][0].as<double>();
  t.inv_idx = d_invidx_.as<int>();
  t.iface_inv = m.iface_inv;
  t.iface_start = m.n_vel_parms;
  t.n_inv = m.n_inv_parms;
  for (int r = 1; r <= 6; ++r) {
    const Region& G = m.reg[r];
    TrRegion& R = t.reg[r];
    R.code = reg_[r].code.as<uint32_t>();
    R.slot_of_node = reg_[r].slot_of_node.as<int>();
    R.r0 = reg_[r].r0.as<int>();
    R.r1 = reg_[r].r1.as<int>();
    R.z_lo = G.z_lo;
    R.H = G.H;
    R.pitch = G.pitch;
    R.itop = G.itop;
    R.ibot = G.ibot;
    R.id = r;
    R.nnode = G.nnode;
  }
  trmodel_ = t;
  return std::string();
}

std::string Engine::trace(const int* src, const int* phase, const double* rx, const double* rz,
                          int npick, double* t_calc, int* valid, long long* nnz, bool rows) {
  cudaSetDevice(device_);
  if (m_.nx == 0) return "no model uploaded";
  if (npick < 0) return "negative pick count";
  const int ns = (int)fields_.size();
  std::vector<TrPick> pk(std::max(npick, 1));
  for (int i = 0; i < npick; ++i) {
    if (src[i] < 0 || src[i] >= ns) return "pick source out of range";
    if (phase[i] < 1 || phase[i] > 5) return "pick phase out of range";
    pk[i].src = src[i];
    pk[i].phase = phase[i];
    pk[i].rx = rx[i];
    pk[i].rz = rz[i];
  }
  std::vector<TrField> tf((size_t)std::max(ns, 1) * 13);
  for (int s = 0; s < ns; ++s)
    for (int k = 1; k <= 12; ++k)
      if (fields_[s][k].solved) {
        tf[(size_t)s * 13 + k].T = fields_[s][k].T.as<double>();
        tf[(size_t)s * 13 + k].G = fields_[s][k].Gout.as<double2>();
      }
  // the entry search's seafloor-node times, once per terminal field of
  // phases 1-3 (tf1, tf3, tf5) of every source
  std::vector<SfJob> jobs;
  {
    const int nsf = m_.nx;
    size_t nj = 0;
    for (int s = 0; s < ns; ++s)
      for (int k : {1, 3, 5})
        if (fields_[s][k].solved) ++nj;
    d_sft_.alloc(std::max<size_t>(nj, 1) * nsf * sizeof(double));
    if (!d_sft_.p) return "device allocation failed (seafloor times)";
    size_t j = 0;
    for (int s = 0; s < ns; ++s)
      for (int k : {1, 3, 5})
        if (fields_[s][k].solved) {
          SfJob J;
          J.T = fields_[s][k].T.as<double>();
          J.reg = kTf[k].reg;
          J.out = d_sft_.as<double>() + j * nsf;
          tf[(size_t)s * 13 + k].sft = J.out;
          jobs.push_back(J);
          ++j;
        }
  }
  std::string e;
  if (!(e = put_vec(d_picks_, pk.data(), (size_t)npick, stream_)).empty()) return e;
  if (!(e = put_vec(d_trfields_, tf.data(), tf.size(), stream_)).empty()) return e;
  if (!jobs.empty()) {
    if (!(e = put_vec(d_sfjobs_, jobs.data(), jobs.size(), stream_)).empty()) return e;
    tr_sf_times(trmodel_, d_sfjobs_.as<SfJob>(), (int)jobs.size(), m_.nx, stream_);
    ++stats_.launches;
    TCK(cudaGetLastError());
  }
  if (!(e = put_vec(d_srcx_, src_x_.data(), (size_t)ns, stream_)).empty()) return e;
  if (!(e = put_vec(d_srcz_, src_z_.data(), (size_t)ns, stream_)).empty()) return e;
  const size_t np = (size_t)std::max(npick, 1);
  d_tcalc_.alloc(np * sizeof(double));
  d_valid_.alloc(np * sizeof(int));
  d_cnt_.alloc((np + 1) * sizeof(unsigned));
  d_off_.alloc((np + 1) * sizeof(unsigned long long));
  d_rowptr_.alloc((np + 1) * sizeof(int));
  d_entry_.alloc(np * 3 * sizeof(double));
  if (!d_tcalc_.p || !d_valid_.p || !d_cnt_.p || !d_off_.p || !d_rowptr_.p || !d_entry_.p)
    return "device allocation failed (picks)";
  // the timing events are released on every return
  struct Events {
    cudaEvent_t a = nullptr, b = nullptr;
    Events() { cudaEventCreate(&a); cudaEventCreate(&b); }
    ~Events() {
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
    }
  } ev;
  cudaEventRecord(ev.a, stream_);
  rows_ = rows ? 0 : -1;
  nnz_ = 0;
  npick_ = -1;   // no rows to hand out unless this trace completes
  if (npick > 0) {
    unsigned* cnt = d_cnt_.as<unsigned>();
    TCK(cudaMemsetAsync(cnt, 0, (np + 1) * sizeof(unsigned), stream_));
    // the pool: entries of a ray as long as its offset and the model's depth
    // twice (four a cell); where that is too little, or memory is short, the
    // rays that count their entries are traced again into one of the right size
    // (sort keys and values; the rays' entries, which the sort's second buffers
    // take the place of, their chunks' owners and counter)
    const CallMem mem = rows ? call_mem() : CallMem();
    struct RowSpace {
      CallBuf keys, vals, ids, pvals, owner, used;
      explicit RowSpace(const CallMem& m) : keys(m), vals(m), ids(m), pvals(m), owner(m), used(m) {}
    } W(mem);
    size_t chunks = 0;
    TrPool pool;
    auto set_pool = [&](size_t n) {
      W.ids.alloc(n * kTrChunk * sizeof(unsigned long long));   // (sort keys later)
      W.pvals.alloc(n * kTrChunk * sizeof(double));
      W.owner.alloc(n * sizeof(uint2));
      const bool ok = W.ids.p && W.pvals.p && W.owner.p;
      pool.ids = W.ids.as<int>();
      pool.vals = W.pvals.as<double>();
      pool.owner = W.owner.as<uint2>();
      pool.nchunks = ok ? (unsigned)std::min({W.ids.bytes / (kTrChunk * 8),
                                              W.pvals.bytes / (kTrChunk * 8),
                                              W.owner.bytes / sizeof(uint2),
                                              (size_t)0x7fffffff}) : 0u;
      return ok;
    };
    if (rows) {
      double len = 0.0;
      for (int i = 0; i < npick; ++i)
        len += std::min(std::fabs(rx[i] - src_x_[src[i]]) / m_.dx, (double)m_.nx) + 2.0 * m_.nz;
      if (!(len >= 0.0)) len = 0.0;   // (a receiver that is not a number)
      chunks = (size_t)(4.0 * len / kTrChunk) + (size_t)npick;
      W.used.alloc(sizeof(unsigned));
      if (!W.used.p) return "device allocation failed (Frechet)";
      const size_t fit = mem.avail / 4 / (kTrChunk * 16 + sizeof(uint2));
      // (no memory for a pool: the rays are counted)
      set_pool(std::min({chunks, fit, (size_t)(0x7fffffffu / kTrChunk) + npick}));
      pool.used = W.used.as<unsigned>();
      TCK(cudaMemsetAsync(W.used.p, 0, sizeof(unsigned), stream_));
    }
    auto launch = [&](bool again) {
      tr_launch(rows ? kTrRows : kTrTimes, trmodel_, d_trfields_.as<TrField>(),
                d_srcx_.as<double>(), d_srcz_.as<double>(), d_picks_.as<TrPick>(), npick,
                d_tcalc_.as<double>(), d_valid_.as<int>(), again, cnt, pool,
                d_entry_.as<double>(), stream_);
      ++stats_.launches;
    };
    launch(false);
    TCK(cudaGetLastError());
    if (!rows) {   // times only (the line search's compute_rms_after_forward)
      TCK(cudaMemcpyAsync(t_calc, d_tcalc_.p, (size_t)npick * 8, cudaMemcpyDeviceToHost, stream_));
      TCK(cudaMemcpyAsync(valid, d_valid_.p, (size_t)npick * 4, cudaMemcpyDeviceToHost, stream_));
      cudaEventRecord(ev.b, stream_);
      TCK(cudaStreamSynchronize(stream_));
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, ev.a, ev.b);
      trace_ms_ = ms;
      npick_ = npick;
      if (nnz) *nnz = 0;
      return std::string();
    }
    auto temp = [&](size_t bytes) {
      d_tmp_.alloc(std::max<size_t>(bytes, 16));
      return d_tmp_.p != nullptr;
    };
    // offsets of each pick's contributions (64-bit: long rays times many picks)
    unsigned long long* off = d_off_.as<unsigned long long>();
    size_t tmp_bytes = 0;
    TCK(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cnt, off, npick + 1, stream_));
    if (!temp(tmp_bytes)) return "device allocation failed (Frechet)";
    TCK(cub::DeviceScan::ExclusiveSum(d_tmp_.p, tmp_bytes, cnt, off, npick + 1, stream_));
    unsigned long long total = 0;
    unsigned used = 0;
    TCK(cudaMemcpyAsync(&total, off + npick, sizeof(total), cudaMemcpyDeviceToHost, stream_));
    TCK(cudaMemcpyAsync(&used, W.used.p, sizeof(used), cudaMemcpyDeviceToHost, stream_));
    TCK(cudaStreamSynchronize(stream_));
    if (total >= 0x7fffffffull) return "too many Frechet contributions for 32-bit CSR";
    if (used > pool.nchunks) {
      if (!set_pool((size_t)total / kTrChunk + npick)) return "device allocation failed (Frechet)";
      TCK(cudaMemsetAsync(W.used.p, 0, sizeof(unsigned), stream_));
      launch(true);
      TCK(cudaGetLastError());
      TCK(cudaMemcpyAsync(&used, W.used.p, sizeof(used), cudaMemcpyDeviceToHost, stream_));
      TCK(cudaStreamSynchronize(stream_));
      if (used > pool.nchunks) return "ray entries out of step with their count";
    }
    const size_t nt = std::max<size_t>((size_t)total, 2);
    W.keys.alloc(nt * 8);
    W.vals.alloc(nt * 8);
    W.ids.alloc(nt * 8);
    W.pvals.alloc(nt * 8);
    if (!W.keys.p || !W.vals.p || !W.ids.p || !W.pvals.p)
      return "device allocation failed (Frechet)";
    cub::DoubleBuffer<unsigned long long> kb(W.keys.as<unsigned long long>(),
                                             W.ids.as<unsigned long long>());
    cub::DoubleBuffer<double> vb(W.vals.as<double>(), W.pvals.as<double>());
    tr_gather(pool, used, d_valid_.as<int>(), cnt, off, kb.Current(), vb.Current(), stream_);
    ++stats_.launches;
    TCK(cudaGetLastError());
    const int n = (int)total;
    int end_bit = 32;
    while (end_bit < 63 && (1ull << (end_bit - 32)) <= (unsigned long long)npick) ++end_bit;
    // stable sort by (pick, parameter): contributions of one entry stay in
    // segment order
    size_t sb = 0;
    TCK(cub::DeviceRadixSort::SortPairs(nullptr, sb, kb, vb, n, 0, end_bit, stream_));
    if (!temp(sb)) return "device allocation failed (Frechet sort)";
    TCK(cub::DeviceRadixSort::SortPairs(d_tmp_.p, sb, kb, vb, n, 0, end_bit, stream_));
    // sum equal keys
    unsigned long long* keys = kb.Alternate();
    double* vals = vb.Alternate();
    int* nruns = W.used.as<int>();
    size_t rb = 0;
    TCK(cub::DeviceReduce::ReduceByKey(nullptr, rb, kb.Current(), keys, vb.Current(), vals, nruns,
                                       ::cuda::std::plus<>{}, n, stream_));
    if (!temp(rb)) return "device allocation failed (Frechet sums)";
    TCK(cub::DeviceReduce::ReduceByKey(d_tmp_.p, rb, kb.Current(), keys, vb.Current(), vals, nruns,
                                       ::cuda::std::plus<>{}, n, stream_));
    int nu = 0;
    TCK(cudaMemcpyAsync(&nu, nruns, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    TCK(cudaStreamSynchronize(stream_));
    // drop zero entries, find each row's start, place the survivors
    int *flag = (int*)kb.Current(), *pos = (int*)vb.Current();   // (nu + 1 <= 2 nt)
    k_keep<<<nu / 256 + 1, 256, 0, stream_>>>(vals, nu, flag);
    ++stats_.launches;
    size_t qb = 0;
    TCK(cub::DeviceScan::ExclusiveSum(nullptr, qb, flag, pos, nu + 1, stream_));
    if (!temp(qb)) return "device allocation failed (Frechet rows)";
    TCK(cub::DeviceScan::ExclusiveSum(d_tmp_.p, qb, flag, pos, nu + 1, stream_));
    k_row_starts<<<npick / 256 + 1, 256, 0, stream_>>>(keys, pos, nu, npick, d_rowptr_.as<int>());
    ++stats_.launches;
    int kept = 0;
    TCK(cudaMemcpyAsync(&kept, pos + nu, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    TCK(cudaStreamSynchronize(stream_));
    d_col_.alloc((size_t)std::max(kept, 1) * 4);
    d_val_.alloc((size_t)std::max(kept, 1) * 8);
    if (!d_col_.p || !d_val_.p) return "device allocation failed (Frechet rows)";
    if (nu > 0)
      k_scatter_rows<<<(nu + 255) / 256, 256, 0, stream_>>>(keys, vals, flag, pos, nu,
                                                            d_col_.as<int>(), d_val_.as<double>());
    ++stats_.launches;
    TCK(cudaGetLastError());
    nnz_ = kept;
    rows_ = npick;
    TCK(cudaMemcpyAsync(t_calc, d_tcalc_.p, (size_t)npick * 8, cudaMemcpyDeviceToHost, stream_));
    TCK(cudaMemcpyAsync(valid, d_valid_.p, (size_t)npick * 4, cudaMemcpyDeviceToHost, stream_));
  }
  cudaEventRecord(ev.b, stream_);
  TCK(cudaStreamSynchronize(stream_));
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, ev.a, ev.b);
  trace_ms_ = ms;
  npick_ = npick;
  if (nnz) *nnz = nnz_;
  return std::string();
}

std::string Engine::trace_entries(double* water_time, double* entry_x, double* entry_z) {
  cudaSetDevice(device_);
  if (npick_ < 0) return "no completed trace";
  if (npick_ == 0) return std::string();
  std::vector<double> e((size_t)npick_ * 3);
  TCK(cudaMemcpyAsync(e.data(), d_entry_.p, e.size() * sizeof(double), cudaMemcpyDeviceToHost,
                      stream_));
  TCK(cudaStreamSynchronize(stream_));
  for (int p = 0; p < npick_; ++p) {
    if (entry_x) entry_x[p] = e[3 * (size_t)p];
    if (entry_z) entry_z[p] = e[3 * (size_t)p + 1];
    if (water_time) water_time[p] = e[3 * (size_t)p + 2];
  }
  return std::string();
}

std::string Engine::frechet_rows(int* row_ptr, int* col, double* val, int base) {
  cudaSetDevice(device_);
  if (npick_ < 0) return "no picks traced";
  if (rows_ < 0) return "no picks traced with Frechet rows (the last trace computed times only)";
  if (row_ptr) {
    std::vector<int> rp(npick_ + 1, 0);
    if (npick_ > 0)
      TCK(cudaMemcpy(rp.data(), d_rowptr_.p, (size_t)(npick_ + 1) * 4, cudaMemcpyDeviceToHost));
    for (int i = 0; i <= npick_; ++i) row_ptr[i] = rp[i] + base;
  }
  if (nnz_ > 0) {
    if (col) {
      TCK(cudaMemcpy(col, d_col_.p, (size_t)nnz_ * 4, cudaMemcpyDeviceToHost));
      if (base == 0)
        for (long long k = 0; k < nnz_; ++k) col[k] -= 1;   // contributions carry 1-based ids
    }
    if (val) TCK(cudaMemcpy(val, d_val_.p, (size_t)nnz_ * 8, cudaMemcpyDeviceToHost));
  }
  return std::string();
}

}  // namespace fmt2d

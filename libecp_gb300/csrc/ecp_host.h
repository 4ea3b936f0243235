// ecp_host.h -- host-side types of the engine (parsed job, device buffers).
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <string>
#include <algorithm>
#include <vector>

#include "ecp_engine.h"
#include "libecp_gb300.h"

namespace ecpgb {

const char *last_error();
void set_error(const char *fmt, ...);

// Job description parsed from getIntegrals-style arrays.
struct Parsed {
  int nAtoms = 0, nShells = 0, nPrims = 0, nCentres = 0, nPairs = 0, dim = 0;
  int maxLECP = 0, maxLBS = 0, largeGridOrder = 1024;
  // derivative order and its shifts: the pair list below holds every shell
  // pair nShift times (pair-major, shift-minor, the reference's callback
  // order), pairShift the shift index of each entry
  int deriv = 0, nShift = 1;
  std::vector<int> ordering;  // a caller's Cartesian order (empty: libint's)
  double tol = 1e-12, acc = 1e-14;
  std::vector<double> geom, primA, primD, termN, termD, termA;
  std::vector<int> shL, shK, shP, shAtom, shAO, shLocal, atomMaxL, atomShell0;
  std::vector<int> ctrAtom, ctrL, ctrT0, ctrNT, termL, chanT0, pairA, pairB, pairShift;
  std::vector<long long> pairOff;
  long long centreStride = 0;
};

int parse_system(const ecpgb_system &s, Parsed &P);

// Derivative shifts (src/libecp.c:240-248): number per order and the pair.
int shift_count(int deriv);
void shift_pair(int deriv, int s, int &shifta, int &shiftb);
// Angular momenta of the blocks a shifted unit hands out: the shifted ones,
// except the order-2 shifts (+1, 0) and (0, +1), whose blocks keep the
// unshifted l (src/libecp.c:356-362).
void shift_block_l(int deriv, int la, int lb, int shifta, int shiftb, int &lpa, int &lpb);
struct TableKey;
TableKey table_key(const Parsed &P);

// The stream on which the calling thread's buffer growth is ordered: with a
// stream set, DBuf grows with cudaFreeAsync / cudaMallocAsync on it, which
// do not wait for the rest of the device (cudaFree does); null: cudaMalloc.
cudaStream_t &alloc_stream();

// Grow-only device buffer.
template <class T>
struct DBuf {
  T *p = nullptr;
  size_t cap = 0;
  bool ensure(size_t n) {
    if (n <= cap) return true;
    cudaStream_t s = alloc_stream();
    if (p) {
      if (s) cudaFreeAsync(p, s);
      else cudaFree(p);
    }
    p = nullptr;
    cap = 0;
    if ((s ? cudaMallocAsync((void **)&p, n * sizeof(T), s) : cudaMalloc((void **)&p, n * sizeof(T))) !=
        cudaSuccess)
      return false;
    cap = n;
    return true;
  }
  // Like ensure, but the memory held stays until the larger one is there.
  bool grow(size_t n) {
    if (n <= cap) return true;
    T *q = nullptr;
    if (cudaMalloc((void **)&q, n * sizeof(T)) != cudaSuccess) return false;
    if (p) cudaFree(p);
    p = q;
    cap = n;
    return true;
  }
  // Releases the memory, ordered on stream s (null: cudaFree).
  void release(cudaStream_t s) {
    if (p) {
      if (s) cudaFreeAsync(p, s);
      else cudaFree(p);
    }
    p = nullptr;
    cap = 0;
  }
  bool upload(const std::vector<T> &v, cudaStream_t s) {
    if (!ensure(v.size() + 1)) return false;
    if (!v.empty() && cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s) != cudaSuccess)
      return false;
    return cudaStreamSynchronize(s) == cudaSuccess;
  }
  ~DBuf() {
    if (p) cudaFree(p);
  }
  DBuf() = default;
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
};

// Pinned host buffers retired while an allocation stream was set: freeing
// one (cudaFreeHost) waits for the whole device, so they are kept here until
// free_retired_pinned() runs at a quiet point (the request server's shutdown).
std::vector<void *> &retired_pinned();
void retire_pinned(void *p);
void free_retired_pinned();

// Grow-only pinned host buffer; grows by at least half its size.
struct PinnedBuf {
  char *p = nullptr;
  size_t cap = 0;
  bool ensure(size_t n) {
    if (n <= cap) return true;
    if (p) {
      if (alloc_stream()) retire_pinned(p);
      else cudaFreeHost(p);
    }
    p = nullptr;
    const size_t want = std::max(n, cap + cap / 2);
    cap = 0;
    if (cudaMallocHost((void **)&p, want) != cudaSuccess) return false;
    cap = want;
    return true;
  }
  ~PinnedBuf() {
    if (p) cudaFreeHost(p);
  }
  PinnedBuf() = default;
  PinnedBuf(const PinnedBuf &) = delete;
  PinnedBuf &operator=(const PinnedBuf &) = delete;
};

// Bytes of each of a job's device buffers, in the order of JobBuffers::each.
constexpr int kJobBufs = 18;
struct JobBytes {
  size_t b[kJobBufs] = {};
  size_t total() const {
    size_t t = 0;
    for (size_t x : b) t += x;
    return t;
  }
};

// Device allocations of one job.
struct JobBuffers {
  DBuf<char> in;
  DBuf<double> radius, utab, uL, F, cgeo, usp, ang, out, mat;
  DBuf<int> gridEnd, win, status, err;
  DBuf<int> live, screenBlocks, liveStart;  // screening stage of the batched path
  DBuf<char> ownScr;             // scratch between the unit stages: a server slot's own,
  DBuf<char> *scr = &ownScr;     // or the one that all jobs of the engine's stream share
  JobPlan plan;
  DBuf<double> sout;       // spherical blocks
  DBuf<long long> sphOff;  // their per-entry offsets
  PinnedBuf pinned, pinnedOut;
  int *pinnedErr = nullptr;
  long long h2dBytes = 0;
  JobBuffers() { cudaMallocHost((void **)&pinnedErr, 4 * sizeof(int)); }
  // Every buffer that staging a job grows.
  template <class F_>
  void each(F_ f) {
    f(in); f(radius); f(utab); f(uL); f(F); f(cgeo); f(usp); f(ang); f(out); f(mat);
    f(gridEnd); f(win); f(status); f(err); f(live); f(screenBlocks); f(liveStart); f(*scr);
  }
  // Device bytes held, and what they will be once a job of `need` is staged (a
  // buffer keeps the larger size).
  size_t device_bytes_with(const JobBytes &need) {
    size_t t = 0;
    int i = 0;
    each([&](auto &d) { t += std::max(d.cap * sizeof(*d.p), need.b[i++]); });
    return t;
  }
  size_t device_bytes() { return device_bytes_with(JobBytes{}); }
  // Grows every buffer to at least its bytes in `need`.
  bool reserve(const JobBytes &need) {
    bool ok = true;
    int i = 0;
    each([&](auto &d) {
      const size_t n = (need.b[i++] + sizeof(*d.p) - 1) / sizeof(*d.p);
      // (resident jobs are planned for the shared scratch as it is)
      ok = ((void *)&d == (void *)scr && scr != &ownScr ? d.grow(n) : d.ensure(n)) && ok;
    });
    return ok;
  }
  // Releases the device buffers (ordered on stream s); they grow again on use.
  void release(cudaStream_t s) {
    each([&](auto &d) { d.release(s); });
    sout.release(s);
    sphOff.release(s);
  }
  ~JobBuffers() {
    if (pinnedErr) cudaFreeHost(pinnedErr);
  }
};

int run_matrix(const ecpgb_system &s, int mode, int rowdim, double *I, ecpgb_info *info);
int run_blocks(const ecpgb_system &s, int mode, double *values, long long *offsets, int *status,
               ecpgb_info *info, Parsed *parsedOut);
int layout(const ecpgb_system &s, long long *nUnits, long long *nValues);
int run_gradient(const ecpgb_system &s, int mode, const double *D, int ldD, double *energy, double *grad);
int layout_sph(const ecpgb_system &s, long long *nUnits, long long *nValues);
int run_blocks_sph(const ecpgb_system &s, int mode, double *values, long long *offsets, int *status);
int cart2sph_table(int l, double *out);
void *job_create(const ecpgb_system &s, int mode);
int job_run(void *j, int nRuns, int flushL2, float *msRun, float *msUnit);
int job_matrix(void *j, int rowdim, double *I);
long long job_units(const void *j, long long *emitted);
int job_launches(const void *j);
void job_free(void *j);
int job_tune(void *j, ecpgb_launch_config *chosen, ecpgb_launch_config *trials, int maxTrials, int *nTrials);
int job_config(void *j, const ecpgb_launch_config *cfg, ecpgb_launch_config *out);
int job_class_config(void *j, int n, int *gcap, int *balance);
int job_use_graph(void *j, int on);
int job_blocks(void *j, double *values, int *status);
int measure_peaks(double *out);

// The engine's lock (serialises every use of the shared __constant__ level
// schedules), and the notice a caller holding it gives after writing those
// schedules itself, so the engine re-uploads its own before its next run.
std::mutex &engine_mutex();
void schedules_overwritten();
// Waits (releasing lk, which holds the engine lock) until no request in
// flight pins the level schedules.
void wait_schedules_unpinned(std::unique_lock<std::mutex> &lk);
int run_matrix_noalloc(const ecpgb_system &s, int rowdim, double *I);

bool valid_mode(int mode);

// ---- internals shared with the request server (ecp_serve.cpp)
struct DevTables;
// Packs P's inputs into B's pinned buffer, copies them to the device on
// `stream` and fills J (B's buffers grow as needed).
// A job's units run in chunks whose scratch stays within scratchCap.  Unit stages
// of the 50-centre cluster, the 83-shell g batch and the 150-shell sweep (ms) with
// 512 MiB: 36.9, 30.5, 47.4; 256: 37.0, 31.2, 48.2; 128: 37.4, 34.6, 51.5; 64: 38.6,
// 38.0, 58.4 (a chunk's last entries leave the GPU idle); 1 and 4 GiB take 0.3 % off.
constexpr size_t kScratchCap = 512ull << 20;
// No cap makes chunks smaller than this (or than one unit): their list and their
// launches would cost more than the scratch they save.
constexpr size_t kScratchFloor = 256ull << 10;
int stage_job(const Parsed &P, const DevTables *T, JobBuffers &B, DevJob &J, int mode, cudaStream_t stream,
              size_t scratchCap = kScratchCap);
// Resets the run's words and launches the pipeline of the mode on `stream`;
// cfg null = the tuned configuration for the job's (l, L).
int run_pipeline(JobBuffers &B, const DevJob &J, int mode, cudaEvent_t u0, cudaEvent_t u1,
                 const FastConfig *cfg, cudaStream_t stream);
// Device bytes of a job of P where at most `budget` may be held, and the scratch
// cap to stage it with; false where its buffers without the unit stages' plan and
// scratch are above the budget.  The scratch takes what the budget leaves, down to
// kScratchFloor or one unit's (which a job that close to the budget holds above it).
bool job_device_bytes(const Parsed &P, int mode, size_t budget, JobBytes *need, size_t *scratchCap);
// With the engine lock held: the tables of the request and, unless requests
// in flight pin other level schedules (returns 4: retry after they finish),
// its schedules made current and pinned.  0 ok, 1 error.
int engine_pin_request(const Parsed &P, int mode, const DevTables **T);
// With the engine lock held: releases one pin.
void engine_unpin_request();
// Server objects (ecp_serve.cpp).
void *server_create(int mode, long long budget, int slots);
long long server_submit(void *sv, const ecpgb_system &s);
int server_poll(void *sv, long long id);
int server_wait(void *sv, long long id, int rowdim, double *I, ecpgb_request_info *info);
int server_stats(void *sv, ecpgb_server_stats *st);
void server_free(void *sv);

}  // namespace ecpgb

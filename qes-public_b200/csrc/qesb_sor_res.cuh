// Types of the resident solve (qesb_sor_res.cu): lambda kept in shared memory
// for a whole solve.
#pragma once
#include "qesb_device.cuh"

namespace qesb {

constexpr int kResMaxThreads = 512;
constexpr int kResPhases = 3;   // start stage, pre-phase, reference loop
constexpr uint32_t kResWaitLimit = 1u << 23;  // polls of a wait before a CTA gives up (seconds)

// One SOR loop of a domain: omega through its table and c1, its stop.
struct ResPhase {
  const float *inv;  // [Z][64] omega / sum of the open faces' coefficients
  double *err;       // [itermax] FP64 max|dlambda| per iteration, zeroed
  SolveState *st;    // zeroed
  double tol;
  float c1;          // 1 - omega
  int itermax;
  int wK;            // window rule's length (0: off)
};

// What the CTAs of a domain share; zeroed before the launch.
struct alignas(128) ResSync {
  unsigned long long bar;  // arrivals at the full barrier
  unsigned long long arr;  // CTAs whose red half-sweep of an iteration is done, summed over the iterations
  unsigned long long pad_[14];
  unsigned cert;           // number of the last iteration proven not to stop
  unsigned beat;           // the first CTA's iteration number, for CTAs of the group that wait for the next domain
  double wacc[4];          // window rule: max|lambda - snapshot|, windows in turn (the first starts from the boundary's)
};

struct ResDomain {
  int X, Y, Z, PQ;
  long CS;
  int nty, ntz;    // tiles along y and z
  int nq4;         // 4-cell groups per colour row
  unsigned magic;  // ceil(2^32 / nq4): division of small numbers by nq4
  int tym, tzm;    // the largest tile's rows and planes
  unsigned epoch;  // mark of the domain's first half-sweep in the exchange buffer
  float *lam;      // [2][CS] split layout; in: the start, out: the result
  const float *R;
  const uint8_t *mask;
  const float *val;  // [6][Z]
  const float *co;   // full coefficients instead of mask and val: [7][2][CS] e f g h m n, omega / (their sum)
  float *snap;       // [2][CS] window snapshot
  uint2 *walls[2];   // [(Y - 2) (Z - 2) 4 nq4] room for each colour's wall cells
  double wtol;
  int nph;
  ResPhase ph[kResPhases];
  ResSync *sync;
  bool alias;        // lam lies in the exchange buffer: read by all CTAs, then the slots cleared, before the first publishes
};

struct ResCtl {
  int queue;  // next domain
  int fault;  // a bounded wait gave up: the results are void
  unsigned long long t0;  // %globaltimer at the start of the launch
};

struct ResArgs {
  const ResDomain *dom;
  int n;                     // domains
  int gsz;                   // CTAs per group: the tiles of the launch's most divided domain
  ResCtl *ctl;
  ulonglong2 *xbuf;          // exchange buffer: [group][colour][CTA][xstride] groups of 4 cells, 32 bytes each
  int xstride;
  unsigned long long *slot;  // [groups] domain handed out by a group's first CTA: (serial << 32) | index
  unsigned wait_limit;
  int smem_floats;           // dynamic shared memory, in floats
};

// Launches the kernel (cooperatively: its CTAs wait on one another) with
// groups * a.gsz CTAs of `threads` threads on s; full: the domains bring their own coefficients (co).
cudaError_t res_launch(const ResArgs &a, bool full, int groups, int threads, cudaStream_t s);

}  // namespace qesb

// Curvilinear WADG solver handle: the reference's stage RK_step_WADG
// (cpp/src/WaveOKL3d.cpp:2111-2185) and its LSRK45 loop (Wave_RK with
// useWADG = 2, cpp/src/WaveOKL3d.cpp:2014-2079), B200 layout:
//
// * elements are renumbered planar first, curved last (host permutation on
//   set/get; the kernel-level entry points keep the reference's numbering);
// * the planar elements [0, KP) advance with the fused affine stage kernel
//   (one pass: volume, surface, WADG projection of p with c^2, LSRK update).
//   For an affine element J is constant, so the reference's J-weighted
//   planar kernels followed by the 1/J update reduce to the unweighted
//   stage with Pq diag(c^2) Vq on p and the identity on u, v, w (Pq Vq = I);
// * the curved elements [KP, K) advance with one fused kernel
//   (k_curved_stage: skew volume + skew surface + 1/J, c^2 WADG update +
//   LSRK update), reading the same old state and writing the same new
//   state buffer, so one stage is two launches and no rhs array exists.
//   The two write disjoint elements, so the curved kernel runs on a second
//   stream beside the planar one (fork / join by events each stage): the
//   planar kernel is bound by its shared-memory pipe, the curved one by
//   latency, and their CTAs share the SMs.
// bbw_curved_steps captures one LSRK45 step per buffer parity in a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "bbwadg.h"
#include "ctx.h"
#include "curved.h"
#include "device_common.cuh"


using namespace bbw;

struct bbw_curved {
  int N = 0, K = 0, Np = 0, KC = 0, KP = 0, device = 0;
  cudaStream_t stream = nullptr, side = nullptr;  // main stream; the curved kernel's
  cudaEvent_t fork = nullptr, join = nullptr;
  bbw_ctx *aff = nullptr;             // fused affine stage of the planar elements
  float *Q[2] = {nullptr, nullptr};   // state buffers (the affine context's when it exists)
  float *res = nullptr;
  int cur = 0;
  std::vector<int> perm;              // new element index -> reference index
  CurvedStageArgs args{};
  CurvedMma mma;                      // matrix form of the curved elements' stage
  int *d_perm = nullptr;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  uint32_t graph_dt_bits[2] = {0, 0};
  std::vector<void *> owned;
};

namespace {

template <class T>
bbw_status own_upload(bbw_curved *h, T **dst, const T *src, size_t n, const char *what) {
  bbw_status s = upload(dst, src, n, what);
  if (s == BBW_OK) h->owned.push_back((void *)*dst);
  return s;
}

template <class T>
const T *own_upload_c(bbw_curved *h, const T *src, size_t n, bbw_status &s) {
  T *d = nullptr;
  if (s == BBW_OK) s = own_upload(h, &d, src, n, "bbw_curved_create: upload");
  return d;
}

// frees one of the handle's buffers
template <class T>
void drop(bbw_curved *h, T *&p) {
  for (size_t i = 0; i < h->owned.size(); ++i)
    if (h->owned[i] == (const void *)p) {
      cudaFree(h->owned[i]);
      h->owned.erase(h->owned.begin() + i);
      break;
    }
  p = nullptr;
}

void release(bbw_curved *h) {
  for (auto &g : h->graph)
    if (g) cudaGraphExecDestroy(g);
  if (h->aff) bbw_destroy(h->aff);
  for (void *p : h->owned) cudaFree(p);
  if (h->fork) cudaEventDestroy(h->fork);
  if (h->join) cudaEventDestroy(h->join);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

// rows of a [K][w] array in the new element order (from position `from`)
template <class T>
std::vector<T> rows(const T *a, const std::vector<int> &perm, size_t w, int from = 0) {
  std::vector<T> out((perm.size() - from) * w);
  for (size_t i = from; i < perm.size(); ++i)
    std::memcpy(&out[(i - from) * w], a + (size_t)perm[i] * w, w * sizeof(T));
  return out;
}

float max_row_sum(const float *A, int nr, int nc) {  // column-major nr x nc
  double m = 0.0;
  for (int i = 0; i < nr; ++i) {
    double s = 0.0;
    for (int j = 0; j < nc; ++j) s += std::fabs((double)A[i + (size_t)j * nr]);
    m = std::max(m, s);
  }
  return (float)m;
}

// split operators and tiled point data of the curved elements' matrix stage;
// leaves h->mma.on false where it does not fit
bbw_status setup_mma(bbw_curved *h, const bbw_curved_desc *d) {
  const CurvedStageArgs &S = h->args;
  CurvedMma &M = h->mma;
  const int Np = h->Np, Nfp = NFP(h->N), Nq = S.Nq, Nfq = S.Nfq, Nr = S.Nr;
  M.KC = S.KC, M.k_off = S.k_off, M.nt = (S.KC + 15) / 16;
  M.nch = (Nq + 15) / 16, M.nchr = (Nr + 15) / 16, M.FC = (Nfq + 15) / 16;
  bbw_status s = curved_mma_prepare(h->N, M);
  if (s == BBW_ERR_UNSUPPORTED) return BBW_OK;
  if (s != BBW_OK) return s;
  const size_t mq = (size_t)Nq * Np, mr = (size_t)Nr * Np;
  const float *hV[4] = {d->Vq, d->Vrq, d->Vsq, d->Vtq}, *hP[4] = {d->Pq, d->Prq, d->Psq, d->Ptq};
  const float sV = split_scale(hV, 1, mq), sD = split_scale(hV + 1, 3, mq);
  const float *pf[1] = {d->Pfq};
  const float sP = std::min(split_scale(hP, 4, mq), split_scale(pf, 1, (size_t)Np * 4 * Nfq));
  const float sF = split_scale(&d->VfqFace, 1, (size_t)Nfq * Nfp);
  const float sVr = split_scale(&d->Vq_reduced, 1, mr), sPr = split_scale(&d->Pq_reduced, 1, mr);
  std::vector<PackRegion> ops;  // of the operators on the device
  const float *V[4] = {S.Vq, S.Vrq, S.Vsq, S.Vtq}, *P[4] = {S.Pq, S.Prq, S.Psq, S.Ptq};
  for (int i = 0; i < 4; ++i) {
    split_rows(ops, V[i], Nq, Np, i == 0 ? sV : sD, M.oV[i], M.oVt[i]);
    split_columns(ops, P[i], Np, Nq, sP, M.oP[i]);
  }
  split_rows(ops, S.VfqFace, Nfq, Nfp, sF, M.oF, M.oFt);
  for (int f = 0; f < 4; ++f) {
    int off = 0;
    split_columns(ops, S.Pfq + (size_t)f * Nfq * Np, Np, Nfq, sP, off);
    if (f == 0) M.oL = off;
  }
  split_rows(ops, S.Vqr, Nr, Np, sVr, M.oVr, M.oVrt);
  split_columns(ops, S.Pqr, Np, Nr, sPr, M.oPr);
  M.oM = ops.back().end();
  M.iV = 1.f / sV, M.iD = 1.f / sD, M.iP = 1.f / sP, M.iF = 1.f / sF, M.iVr = 1.f / sVr,
  M.iPr = 1.f / sPr;
  M.vnorm = max_row_sum(d->Vq, Nq, Np), M.rnorm = max_row_sum(d->Vq_reduced, Nr, Np);
  M.fnorm = max_row_sum(d->VfqFace, Nfq, Nfp);
  M.dnorm = std::max(max_row_sum(d->Vrq, Nq, Np),
                     std::max(max_row_sum(d->Vsq, Nq, Np), max_row_sum(d->Vtq, Nq, Np)));
  uint4 *dops = nullptr;
  float *gq = nullptr, *fq = nullptr, *jq = nullptr, *bound = nullptr;
  const size_t nt = M.nt;
  const float *none = nullptr;
  if ((s = own_upload(h, &dops, (const uint4 *)nullptr, (size_t)M.oM / 4 * 5, "bbw_curved_create")) !=
          BBW_OK ||
      (s = pack_operators(ops, dops, dops + M.oM)) != BBW_OK ||
      (s = own_upload(h, &gq, none, nt * M.nch * 10 * 256, "bbw_curved_create")) != BBW_OK ||
      (s = own_upload(h, &fq, none, nt * 4 * M.FC * 4 * 256, "bbw_curved_create")) != BBW_OK ||
      (s = own_upload(h, &jq, none, nt * M.nchr * 2 * 256, "bbw_curved_create")) != BBW_OK ||
      (s = own_upload(h, &bound, none, (size_t)M.KC * 8, "bbw_curved_create")) != BBW_OK ||
      (s = curved_mma_points(S, M, gq, fq, jq, bound)) != BBW_OK)
    return s;
  M.ops = dops, M.gq = gq, M.fq = fq, M.jq = jq, M.bound = bound;
  M.Fmask = S.Fmask, M.vmapP = S.vmapP;
  M.on = true;
  return BBW_OK;
}

bbw_status stage(bbw_curved *h, float fa, float fb, float fdt) {
  const float *Qin = h->Q[h->cur];
  float *Qout = h->Q[h->cur ^ 1];
  const bool both = h->KP > 0 && h->KC > 0;
  cudaStream_t cst = both ? h->side : h->stream;
  bbw_status s = BBW_OK;
  if (both) {  // fork: the curved kernel waits for everything before this stage
    cudaError_t e = cudaEventRecord(h->fork, h->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(h->side, h->fork, 0);
    s = set_cuda_error(e, "curved stage: fork");
  }
  if (s == BBW_OK && h->KP > 0)
    s = launch_stage(h->aff, Qin, Qout, h->res, fa, fb, fdt, 0.f, h->stream);
  if (s == BBW_OK && h->KC > 0) {
    if (h->mma.on) {
      CurvedMma A = h->mma;
      A.fa = fa, A.fb = fb, A.fdt = fdt;
      s = curved_mma_stage(h->N, A, Qin, Qout, h->res, cst);
    } else {
      CurvedStageArgs A = h->args;
      A.fa = fa, A.fb = fb, A.fdt = fdt;
      s = curved_stage(h->N, A, Qin, Qout, h->res, cst);
    }
  }
  if (both) {  // join: the next stage reads what both wrote (always joined)
    cudaError_t e = cudaEventRecord(h->join, h->side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(h->stream, h->join, 0);
    if (s == BBW_OK) s = set_cuda_error(e, "curved stage: join");
  }
  if (s == BBW_OK) h->cur ^= 1;
  return s;
}

void drop_graphs(bbw_curved *h) {
  for (int i = 0; i < 2; ++i) {
    if (h->graph[i]) cudaGraphExecDestroy(h->graph[i]);
    h->graph[i] = nullptr;
  }
}

}  // namespace

extern "C" bbw_status bbw_curved_create(const bbw_curved_desc *d, int device, bbw_curved **out) {
  if (!out || !d) return set_error(BBW_ERR_ARG, "bbw_curved_create: NULL argument");
  *out = nullptr;
  const int N = d->N, K = d->K;
  if (N < 1 || N > BBW_MAX_N) return set_error(BBW_ERR_UNSUPPORTED, "bbw_curved_create: N");
  const int Np = NP(N), Nfp = NFP(N), NF = 4 * Nfp;
  if (K < 1 || d->Nq < Np || d->Nfq < 1 || d->Nq_reduced < 1 || d->KCurved < 0 ||
      d->KPlanar < 0 || d->KCurved + d->KPlanar != K || (long long)K * 4 * Np >= (1LL << 31))
    return set_error(BBW_ERR_ARG, "bbw_curved_create: bad sizes");
  const void *req[] = {d->vgeo, d->fgeo, d->Jplanar, d->Fmask, d->vmapP, d->Jq_reduced, d->c2q,
                       d->Dr, d->Ds, d->Dt, d->LIFT, d->Vq_reduced, d->Pq_reduced};
  for (const void *p : req)
    if (!p) return set_error(BBW_ERR_ARG, "bbw_curved_create: missing array");
  if (d->KCurved > 0) {
    const void *creq[] = {d->KlistCurved, d->vgeoq, d->Jq, d->fgeoq, d->Vq, d->Vrq, d->Vsq,
                          d->Vtq, d->Pq, d->Prq, d->Psq, d->Ptq, d->VfqFace, d->Pfq};
    for (const void *p : creq)
      if (!p) return set_error(BBW_ERR_ARG, "bbw_curved_create: missing curved-element array");
  }
  if (d->KPlanar > 0 && !d->KlistPlanar)
    return set_error(BBW_ERR_ARG, "bbw_curved_create: missing planar list");
  // every element in exactly one list: planar first, then curved
  std::vector<int> perm, inv(K, -1);
  for (int pass = 0; pass < 2; ++pass) {
    const int n = pass ? d->KCurved : d->KPlanar;
    const int *L = pass ? d->KlistCurved : d->KlistPlanar;
    for (int i = 0; i < n; ++i) {
      if (L[i] < 0 || L[i] >= K || inv[L[i]] >= 0)
        return set_error(BBW_ERR_ARG, "bbw_curved_create: element lists must partition 0..K-1");
      inv[L[i]] = (int)perm.size();
      perm.push_back(L[i]);
    }
  }
  for (int i = 0; i < NF; ++i)
    if (d->Fmask[i] < 0 || d->Fmask[i] >= Np)
      return set_error(BBW_ERR_ARG, "bbw_curved_create: Fmask entry out of range");
  std::vector<int> vmapP((size_t)K * NF);
  for (int i = 0; i < K; ++i)
    for (int m = 0; m < NF; ++m) {
      const int v = d->vmapP[(size_t)perm[i] * NF + m];
      if (v < 0 || v >= K * 4 * Np || v % (4 * Np) >= Np)
        return set_error(BBW_ERR_ARG, "bbw_curved_create: vmapP entry out of range");
      vmapP[(size_t)i * NF + m] = inv[v / (4 * Np)] * 4 * Np + v % (4 * Np);
    }
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_create: device");
  if (device < 0 || device >= ndev)
    return set_error(BBW_ERR_ARG, "bbw_curved_create: no such device");
  DeviceGuard dg(device);  // the caller's current device is restored on return
  bbw_curved *h = new bbw_curved;
  h->N = N, h->K = K, h->Np = Np, h->KC = d->KCurved, h->KP = d->KPlanar, h->device = device;
  h->perm = perm;
  e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    release(h);
    return set_cuda_error(e, "bbw_curved_create: stream");
  }
  const size_t ns = (size_t)K * 4 * Np;
  const int Nq = d->Nq, Nfq = d->Nfq, Nr = d->Nq_reduced, KP = d->KPlanar;
  bbw_status s = BBW_OK;
  std::vector<float> c2 = rows(d->c2q, perm, Nr);
  if (KP > 0) {  // fused affine stage over the planar prefix
    std::vector<float> vgeo = rows(d->vgeo, perm, 9), fgeo = rows(d->fgeo, perm, 16);
    bbw_mesh_desc md{N, K, Nr, vgeo.data(), fgeo.data(), d->Fmask, vmapP.data(), c2.data(),
                     nullptr};
    bbw_ops_desc od{};
    od.Dr = d->Dr, od.Ds = d->Ds, od.Dt = d->Dt, od.LIFT = d->LIFT;
    od.Vq = d->Vq_reduced, od.Pq = d->Pq_reduced;
    s = bbw_create(&md, &od, BBW_NODAL, BBW_BC_PRESSURE_RELEASE, &h->aff);
    // its form by the planar elements alone.  At N = 4 the group form holds the SMs
    // that the thread-per-output kernel runs on beside it (KC = 720: 34.9 us per
    // stage, 29.9 with the CTA-wide stage)
    if (s == BBW_OK && KP < K) s = bbw_set_compute_range(h->aff, KP);
    if (s == BBW_OK) s = bbw_set_whole_mesh(h->aff, KP);
    if (s == BBW_OK && N == 4 && !curved_mma_preferred(N, d->KCurved)) h->aff->cta_form = true;
    if (s == BBW_OK) h->Q[0] = h->aff->Q[0], h->Q[1] = h->aff->Q[1], h->res = h->aff->res;
  } else {
    if (s == BBW_OK) s = own_upload(h, &h->Q[0], (const float *)nullptr, ns, "bbw_curved_create");
    if (s == BBW_OK) s = own_upload(h, &h->Q[1], (const float *)nullptr, ns, "bbw_curved_create");
    if (s == BBW_OK) s = own_upload(h, &h->res, (const float *)nullptr, ns, "bbw_curved_create");
  }
  if (d->KCurved > 0) {  // compact rows of the curved tail
    CurvedStageArgs &A = h->args;
    A.KC = d->KCurved, A.k_off = KP, A.Nq = Nq, A.Nfq = Nfq, A.Nr = Nr;
    const size_t nq = Nq, nr = Nr, nf = Nfq;
    std::vector<float> t;
    t = rows(d->vgeoq, perm, 9 * nq, KP), A.vgeoq = own_upload_c(h, t.data(), t.size(), s);
    t = rows(d->Jq, perm, nq, KP), A.Jq = own_upload_c(h, t.data(), t.size(), s);
    t = rows(d->fgeoq, perm, 16 * nf, KP), A.fgeoq = own_upload_c(h, t.data(), t.size(), s);
    t = rows(d->Jq_reduced, perm, nr, KP), A.Jr = own_upload_c(h, t.data(), t.size(), s);
    A.c2q = own_upload_c(h, c2.data() + (size_t)KP * Nr, (size_t)d->KCurved * Nr, s);
    const size_t mq = nq * Np, mr = nr * Np;
    A.Vq = own_upload_c(h, d->Vq, mq, s), A.Vrq = own_upload_c(h, d->Vrq, mq, s);
    A.Vsq = own_upload_c(h, d->Vsq, mq, s), A.Vtq = own_upload_c(h, d->Vtq, mq, s);
    A.Pq = own_upload_c(h, d->Pq, mq, s), A.Prq = own_upload_c(h, d->Prq, mq, s);
    A.Psq = own_upload_c(h, d->Psq, mq, s), A.Ptq = own_upload_c(h, d->Ptq, mq, s);
    A.VfqFace = own_upload_c(h, d->VfqFace, nf * Nfp, s);
    A.Pfq = own_upload_c(h, d->Pfq, (size_t)Np * 4 * nf, s);
    A.Vqr = own_upload_c(h, d->Vq_reduced, mr, s), A.Pqr = own_upload_c(h, d->Pq_reduced, mr, s);
    A.Fmask = own_upload_c(h, d->Fmask, (size_t)NF, s);
    A.vmapP = own_upload_c(h, vmapP.data(), vmapP.size(), s);
    if (s == BBW_OK && curved_mma_preferred(N, d->KCurved)) {
      const size_t kept = h->owned.size();
      s = setup_mma(h, d);
      if (s == BBW_ERR_NOMEM) {  // no room beside the compact rows: the thread-per-output kernel
        cudaGetLastError();
        for (; h->owned.size() > kept; h->owned.pop_back()) cudaFree(h->owned.back());
        h->mma = CurvedMma();
        s = BBW_OK;
      }
      if (h->mma.on)  // its tiles hold the same point data, its operators are split
        for (const float **p : {&A.vgeoq, &A.Jq, &A.fgeoq, &A.Jr, &A.c2q, &A.Vq, &A.Vrq, &A.Vsq, &A.Vtq,
                                &A.Pq, &A.Prq, &A.Psq, &A.Ptq, &A.VfqFace, &A.Pfq, &A.Vqr, &A.Pqr})
          drop(h, *p);
    }
  }
  if (s == BBW_OK) s = own_upload(h, &h->d_perm, perm.data(), perm.size(), "bbw_curved_create");
  // one stage on the zero state (it stays zero) sets the kernels' launch
  // attributes outside any later graph capture
  if (s == BBW_OK) s = stage(h, 0.f, 0.f, 0.f);
  if (s == BBW_OK) s = set_cuda_error(cudaStreamSynchronize(h->stream), "bbw_curved_create");
  if (s != BBW_OK) {
    release(h);
    return s;
  }
  h->cur = 0;
  *out = h;
  return BBW_OK;
}

extern "C" bbw_status bbw_curved_destroy(bbw_curved *h) {
  if (!h) return BBW_OK;
  DeviceGuard dg(h->device);
  cudaStreamSynchronize(h->stream);
  drop_graphs(h);
  release(h);
  return BBW_OK;
}

// rows of w4 float4: to_new: out[i] = in[perm[i]], else out[perm[i]] = in[i]
__global__ void k_permute_rows(int K, int w4, bool to_new, const int *__restrict__ perm,
                               const float4 *__restrict__ in, float4 *__restrict__ out) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long i = j / w4;
  if (i >= K) return;
  const long long c = j - i * w4, o = (long long)__ldg(perm + i) * w4 + c;
  if (to_new) out[j] = in[o];
  else out[o] = in[j];
}

// host [K][4][Np] in the reference's element order <-> device buffer, permuted on
// the device through the next state's buffer, which every stage writes in full.
// Permuting on the host and copying through pageable memory took 9 ms of the 28
// ms of 20 steps at N = 3, K = 82944 (26 MB each way).
static bbw_status copy_state(bbw_curved *h, float *dev, const float *src, float *dst,
                             const char *what) {
  if (!h || (!src && !dst)) return set_error(BBW_ERR_ARG, what);
  const size_t n = (size_t)h->K * 4 * h->Np;
  float *tmp = h->Q[h->cur ^ 1];
  const int blocks = (int)(((size_t)h->K * h->Np + 255) / 256);
  const float4 *in = reinterpret_cast<const float4 *>(src ? tmp : dev);
  float4 *out = reinterpret_cast<float4 *>(src ? dev : tmp);
  cudaError_t e = cudaSuccess;
  if (src) e = cudaMemcpyAsync(tmp, src, n * sizeof(float), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess) {
    k_permute_rows<<<blocks, 256, 0, h->stream>>>(h->K, h->Np, src != nullptr, h->d_perm, in, out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && dst)
    e = cudaMemcpyAsync(dst, tmp, n * sizeof(float), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  return set_cuda_error(e, what);
}

extern "C" bbw_status bbw_curved_set_state(bbw_curved *h, const float *Q) {
  DeviceGuard dg(h ? h->device : -1);
  bbw_status s = copy_state(h, h ? h->Q[h->cur] : nullptr, Q, nullptr, "bbw_curved_set_state");
  if (s != BBW_OK) return s;
  const size_t n = (size_t)h->K * 4 * h->Np * sizeof(float);
  cudaError_t e = cudaMemsetAsync(h->res, 0, n, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  return set_cuda_error(e, "bbw_curved_set_state");
}

extern "C" bbw_status bbw_curved_get_state(bbw_curved *h, float *Q) {
  DeviceGuard dg(h ? h->device : -1);
  return copy_state(h, h ? h->Q[h->cur] : nullptr, nullptr, Q, "bbw_curved_get_state");
}

extern "C" bbw_status bbw_curved_get_residual(bbw_curved *h, float *r) {
  DeviceGuard dg(h ? h->device : -1);
  return copy_state(h, h ? h->res : nullptr, nullptr, r, "bbw_curved_get_residual");
}

extern "C" bbw_status bbw_curved_stage(bbw_curved *h, float fa, float fb, float fdt) {
  DeviceGuard dg(h ? h->device : -1);
  if (!h) return set_error(BBW_ERR_ARG, "bbw_curved_stage: NULL handle");
  return stage(h, fa, fb, fdt);
}

extern "C" bbw_status bbw_curved_steps(bbw_curved *h, float dt, int nsteps) {
  DeviceGuard dg(h ? h->device : -1);
  if (!h || nsteps < 0) return set_error(BBW_ERR_ARG, "bbw_curved_steps: bad argument");
  uint32_t bits;
  std::memcpy(&bits, &dt, 4);
  for (int step = 0; step < nsteps; ++step) {
    const int par = h->cur;
    if (!h->graph[par] || h->graph_dt_bits[par] != bits) {
      if (h->graph[par]) cudaGraphExecDestroy(h->graph[par]);
      h->graph[par] = nullptr;
      cudaGraph_t g;
      cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_steps: capture");
      bbw_status s = BBW_OK;
      for (int i = 0; i < 5 && s == BBW_OK; ++i)
        s = stage(h, (float)kRK4A[i], (float)kRK4B[i], dt);
      e = cudaStreamEndCapture(h->stream, &g);
      h->cur = par;  // capture recorded the launches without running them
      if (s != BBW_OK) {
        if (e == cudaSuccess) cudaGraphDestroy(g);
        return s;
      }
      if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_steps: end capture");
      e = cudaGraphInstantiate(&h->graph[par], g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_steps: instantiate");
      h->graph_dt_bits[par] = bits;
    }
    cudaError_t e = cudaGraphLaunch(h->graph[par], h->stream);
    if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_steps: launch");
    h->cur ^= 1;  // five stages swap the buffers an odd number of times
  }
  return BBW_OK;
}

extern "C" bbw_status bbw_curved_sync(bbw_curved *h) {
  DeviceGuard dg(h ? h->device : -1);
  if (!h) return set_error(BBW_ERR_ARG, "bbw_curved_sync: NULL handle");
  return set_cuda_error(cudaStreamSynchronize(h->stream), "bbw_curved_sync");
}

extern "C" void *bbw_curved_stream(bbw_curved *h) { return h ? (void *)h->stream : nullptr; }

extern "C" bbw_status bbw_curved_autotune(bbw_curved *h, float dt, int stages, int *config) {
  DeviceGuard dg(h ? h->device : -1);
  if (!h || !(dt > 0.f) || stages < 1)
    return set_error(BBW_ERR_ARG, "bbw_curved_autotune: bad argument");
  if (config) *config = 0;
  if (!h->aff) return BBW_OK;  // no planar element: nothing to choose
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->side);
  if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_autotune");
  // the captured steps hold the planar variant's operator buffer, which
  // bbw_set_config frees: recapture after tuning
  drop_graphs(h);
  const size_t n = (size_t)h->K * 4 * h->Np;
  float *saveQ = nullptr, *saveR = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto cleanup = [&]() {
    cudaFree(saveQ), cudaFree(saveR);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  };
  e = cudaMalloc(&saveQ, n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&saveR, n * sizeof(float));
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  const int cur0 = h->cur;
  if (e == cudaSuccess)
    e = cudaMemcpy(saveQ, h->Q[cur0], n * sizeof(float), cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(saveR, h->res, n * sizeof(float), cudaMemcpyDeviceToDevice);
  if (e != cudaSuccess) {
    cleanup();
    return set_cuda_error(e, "bbw_curved_autotune: scratch");
  }
  float best_ms = 0.f;
  int best = -1;
  bbw_status s = BBW_OK;
  std::vector<int> codes = {kWarpConfig, kGroupConfig};
  for (int e16 = 0; e16 < 2; ++e16)
    for (int W = 8; W <= 16; W += 8)
      for (int v = 0; v < 4; ++v)
        codes.push_back(W | (v < 2 ? 1 << 8 : 0) | (v % 2 == 0 ? 1 << 9 : 0) | e16 << 10);
  for (int code : codes) {
      if (s != BBW_OK) break;
      if (bbw_set_config(h->aff, code) != BBW_OK) continue;  // does not fit
      for (int i = 0; i < 2 && s == BBW_OK; ++i) s = stage(h, 0.f, (float)kRK4B[0], dt);
      if (s == BBW_OK) e = cudaEventRecord(e0, h->stream);
      for (int i = 0; i < stages && s == BBW_OK && e == cudaSuccess; ++i)
        s = stage(h, (float)kRK4A[i % 5], (float)kRK4B[i % 5], dt);
      if (s == BBW_OK && e == cudaSuccess) e = cudaEventRecord(e1, h->stream);
      if (s == BBW_OK && e == cudaSuccess) e = cudaEventSynchronize(e1);
      if (s == BBW_OK && e != cudaSuccess) s = set_cuda_error(e, "bbw_curved_autotune: timing");
      float ms = 0.f;
      if (s == BBW_OK) cudaEventElapsedTime(&ms, e0, e1);
      if (s == BBW_OK && (best < 0 || ms < best_ms)) best = code, best_ms = ms;
    }
  // the state and residual as they were, the fastest variant kept
  h->cur = cur0;
  e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->side);
  if (e == cudaSuccess)
    e = cudaMemcpy(h->Q[cur0], saveQ, n * sizeof(float), cudaMemcpyDeviceToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(h->res, saveR, n * sizeof(float), cudaMemcpyDeviceToDevice);
  cleanup();
  if (s != BBW_OK) return s;
  if (e != cudaSuccess) return set_cuda_error(e, "bbw_curved_autotune: restore");
  if (best < 0) return set_error(BBW_ERR_UNSUPPORTED, "bbw_curved_autotune: no variant fits");
  if ((s = bbw_set_config(h->aff, best)) != BBW_OK) return s;
  if (config) *config = best;
  return BBW_OK;
}

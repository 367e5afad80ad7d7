// md_ctx.cu -- the C ABI (include/md_gb300.h): context, device buffers,
// step orchestration and CUDA-graph replay of one time step.
//
// One step on the device (RunSimulation loop body, src/simulation.cpp:469-518):
//   cells (a) -> real space full (b) -> k space full (c) -> Heun stage 1 (d)
//   -> real space field (b) -> k space field (c) -> Heun stage 2 (d) -> records
// The step reads its time and step number from device memory, so the same
// captured graph is replayed for every step.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "../../include/md_gb300.h"
#include "md_common.cuh"
#include "md_host.h"
#include "md_kernels.h"
#include "md_ctx_internal.h"

namespace {

std::mutex g_err_mu;
std::string g_err;
int g_err_status = 0;

}  // namespace

// Records the boundary event `k` when profiling.
static void mark(md_ctx* c, int k) {
  if (c->prof) cudaEventRecordWithFlags(c->ev[k], c->stream, cudaEventRecordExternal);
}

// ------------------------------------------------------------- helpers

int set_err(md_ctx* c, int status, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (c) {
    c->err = buf;
    c->err_status = status;
  }
  std::lock_guard<std::mutex> lk(g_err_mu);
  g_err = buf;
  g_err_status = status;
  return status;
}


// Device memory of a context comes from the device's default memory pool,
// ordered on the context's stream: freeing (cudaFreeAsync) does not wait for
// the whole GPU as cudaFree does, so contexts that finish while a batch runs
// cost the request loop little, and their memory serves the next contexts.
// The pool keeps freed memory for reuse (release threshold raised once per
// device) instead of returning it to the driver at every synchronisation.
void pool_keep(int device) {
  static std::mutex mu;
  static std::vector<int> done;
  std::lock_guard<std::mutex> lk(mu);
  if (std::find(done.begin(), done.end(), device) != done.end()) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
    uint64_t keep = ~0ull;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  done.push_back(device);
}

int dalloc_raw(md_ctx* c, void** p, size_t bytes) {
  void* q = nullptr;
  if (bytes == 0) bytes = 16;
  cudaError_t e = cudaMallocAsync(&q, bytes, c->stream);
  // the allocation is complete before any stream, or a synchronous copy,
  // touches it
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess)
    return set_err(c, MD_ERR_NOMEM, "device allocation (%zu bytes) failed: %s", bytes, cudaGetErrorString(e));
  c->allocs.push_back(q);
  c->alloc_bytes.push_back(bytes);
  c->bytes += (int64_t)bytes;
  *p = q;
  return MD_OK;
}

void dfree(md_ctx* c, void* p) {
  if (!p) return;
  auto it = std::find(c->allocs.begin(), c->allocs.end(), p);
  if (it != c->allocs.end()) {
    const size_t k = (size_t)(it - c->allocs.begin());
    c->bytes -= (int64_t)c->alloc_bytes[k];
    c->alloc_bytes.erase(c->alloc_bytes.begin() + (ptrdiff_t)k);
    c->allocs.erase(it);
  }
  cudaFreeAsync(p, c->stream);  // after the context's queued work (its side stream joins it)
}

bool fp64(const md_ctx* c) { return c->prec == MD_PREC_FP64; }
size_t tsz(const md_ctx* c) { return fp64(c) ? 8 : 4; }

void invalidate_graph(md_ctx* c) {
  if (c->gexec) cudaGraphExecDestroy(c->gexec);
  if (c->graph) cudaGraphDestroy(c->graph);
  if (c->gexec_n) cudaGraphExecDestroy(c->gexec_n);
  if (c->graph_n) cudaGraphDestroy(c->graph_n);
  c->gexec = c->gexec_n = nullptr;
  c->graph = c->graph_n = nullptr;
  c->graph_valid = false;
  c->replays = 0;
}

SortedView sorted_view(md_ctx* c) {
  SortedView s;
  s.xf = c->xf;
  s.xi = c->xi4;
  s.xd = c->xd;
  s.mu = c->mu;
  s.cell = c->scell;
  s.perm = c->perm;
  s.rank = c->rank;
  s.cell_start = c->cell_start;
  return s;
}

double B_unit(const md_ctx* c) { return c->cfg.facEwald * c->props.muMax / std::pow(c->L, 3.0); }
double F_unit(const md_ctx* c) { return c->cfg.facEwald * c->props.muMax * c->props.muMax / std::pow(c->L, 4.0); }

RealParams real_params(md_ctx* c, void* B, void* F, void* ov) {
  RealParams p{};
  const md_config& g = c->cfg;
  const double L = c->L, a = c->alpha * L, rcb = c->rc / L;
  p.n = (int)c->n;
  p.gtab = c->gtab;
  p.etab = c->etab;
  p.grid = c->grid;
  p.alpha = a;
  p.rc = rcb;
  p.rc2 = rcb * rcb;
  p.pk = make_pair_consts(a, 2.0 * a * g.irPi, 1e-10 / L, p.rc2);
  p.c2a = 2.0 * a * g.irPi;
  p.al2 = a * a;
  p.al4 = p.al2 * p.al2;
  p.cont_eps = 1e-10 / L;
  p.coat = (int)g.ENABLE_COATING_POT;
  const double Fu = F_unit(c);
  p.rcut_sr2 = g.ENABLE_COATING_POT ? std::pow(c->props.rCutSR / L, 2.0) : -1.0;
  p.eff_len = g.effLenSurfMol / L;
  p.ster = g.sterRepFac * L * L / Fu;
  p.elec = g.electrostatRepFac * L / Fu;
  p.kappa = g.kappa * L;
  p.vdw = g.hamaker / (L * Fu);
  p.rMag_u = c->rMag_u;
  p.s = sorted_view(c);
  p.B = B;
  p.F = F;
  p.ov = ov;
  p.Ppart = c->Ppart;
  p.err = &c->sc->err;
  const double rl = rcb * (1.0 + c->skin_frac);
  p.rl2 = rl * rl;
  p.nbr = c->nbr;
  p.nbr_cnt = c->nbr_cnt;
  p.nbr_off = c->nbr_off;
  p.nbr_cap = c->nbr_cap;
  p.nbr_share = (int)(std::min<long long>(c->nbr_cap, 0x7fffffff) / c->n);
  p.flags = &c->sc->flags;
  if (strong_active(c)) {
    p.strong = 1;
    p.strong_w4sq = c->strong_w4sq;
    p.snbr = c->snbr;
    p.snbr_cnt = c->snbr_cnt;
    p.snbr_off = c->snbr_off;
    p.scap = c->scap;
    p.svals = B == c->Br2 ? c->svals2 : c->svals;
    if (B != c->Br2) {  // full evaluation: the master moments
      p.smm = c->mm;
      p.smag = c->magMom_u;
    }
  }
  return p;
}

static MeshGrid mesh_grid(const md_ctx* c) {
  MeshGrid m{};
  if (c->gm_M == 0) return m;
  m.M = c->gm_M;
  m.ncx = c->grid.ncx;
  m.nbrick = md::mesh_bricks(c->gm_M);
  m.nitem = md::mesh_items(c->gm_M);
  // half the skin since the build, and rounding
  m.reach = (float)(0.5 * c->cell_skin * c->rc / c->L * (1.0 + 1e-5) + 2e-6);
  m.plan = c->gm_plan;
  return m;
}

CellParams cell_params(md_ctx* c) {
  CellParams p{};
  p.n = (int)c->n;
  p.invL = 1.0 / c->L;
  p.grid = c->grid;
  p.half_skin = (float)(0.5 * c->skin_frac * c->rc / c->L);
  p.pos = c->pos;
  p.mm = c->mm;
  p.magMom_u = c->magMom_u;
  p.rMag_u = c->rMag_u;
  p.cellOf = c->cellOf;
  p.count = c->count;
  p.tmp = c->tmp;
  p.s = sorted_view(c);
  p.xbuild = c->xbuild;
  p.flags = &c->sc->flags;
  p.mesh = mesh_grid(c);
  return p;
}

ObsParams obs_params(md_ctx* c, double dt) {
  ObsParams o{};
  o.nblk_int = int_blocks((int)c->n);
  o.obs_part = c->obs_part;
  o.p_scale = c->L * F_unit(c) / (2.0 * std::pow(c->L, 3.0));
  o.inv_n = 1.0 / (double)c->n;
  o.dt = dt;
  o.time = &c->sc->time;
  o.stepno = &c->sc->step;
  o.records = c->records;
  o.nrec = &c->sc->nrec;
  o.cap = c->rec_cap;
  o.err = &c->sc->err;
  o.flags = &c->sc->flags;
  o.status = nullptr;
  return o;
}

KParams k_params(md_ctx* c, void* B, void* F) {
  KParams p{};
  p.n = (int)c->n;
  p.kc = (int)c->kc;
  p.nseg = (int)c->klist.seg.size();
  p.nk = c->klist.nk;
  p.chunk = c->chunk;
  p.nchunk = c->nchunk;
  p.two_pi = 2.0 * c->cfg.my_pi;
  p.seg = c->kseg;
  p.koff = c->koff;
  p.ek = c->ek;
  p.rseg = c->rseg;
  p.rowpos = c->rowpos;
  p.chunks = c->chunks;
  p.nchk = c->klist.nchk;
  p.Spart = c->Spart;
  p.musum_part = c->musum_part;
  p.musum = c->sc->musum;
  p.eS = c->eS;
  p.S = c->Sfull;
  p.tab = c->ptab;
  p.cflux = 4.0 * c->cfg.my_pi;
  p.cforce = 8.0 * c->cfg.my_pi * c->cfg.my_pi;
  p.s = sorted_view(c);
  p.B = B;
  p.F = F;
  p.tc_rows = c->tc_rows;
  p.tc_mt = c->tcs.mt;
  p.tc_ns = c->tcs.ns;
  p.tc_kp = c->tcs.kp;
  p.tc_rt = F ? c->tcs.rt_full : c->tcs.rt_field;
  p.tc_nt = F ? c->tcs.nt_full : c->tcs.nt_field;
  p.tc_nst = c->tcs.nst;
  p.tc_chunk = c->tcs.chunk;
  p.tc_nchunk = c->tcs.nchunk;
  p.tc_row = c->tc_row;
  p.tc_rowd = c->tc_rowd;
  p.tc_kmap = c->tc_kmap;
  p.tc_part = c->tc_part;
  p.tc_w = F ? c->tc_wfull : c->tc_wfield;
  p.tc_bimg = c->tc_bimg;
  p.tc_tblk = c->tc_tblk;
  p.tc_scat_smem = c->tcs.scat_smem;
  p.tc_yz = c->tcs.yz;
  p.tc_sfa = c->tcs.sfa;
  p.tc_sfb = c->tcs.sfb;
  p.rw_T = c->rw_T;
  p.rw_R = c->rw_R;
  p.rw_nblk = c->rws.nblk;
  p.rw_threads = c->rws.threads;
  p.rw_chunk = c->rws.chunk;
  p.rw_nchunk = c->rws.nchunk;
  p.rw_np = c->rws.np;
  p.rw_task = c->rw_task;
  p.rw_kidx = c->rw_kidx;
  p.rw_row = c->rw_row;
  p.rw_rowt = c->rw_rowt;
  p.rw_ad = c->rw_ad;
  p.gm_M = c->gm_M;
  const MeshGrid m = mesh_grid(c);
  p.gm_nbrick = m.nbrick;
  p.gm_nitem = m.nitem;
  p.gm_ncx = m.ncx;
  p.gm_reach = m.reach;
  p.gm_coef = c->gm_coef;
  p.gm_fac = c->gm_fac;
  p.gm_tw = c->gm_tw;
  p.gm_part = c->gm_part;
  p.gm_z = c->gm_z;
  p.gm_y = c->gm_y;
  p.gm_t = c->gm_t;
  p.gm_b = c->gm_b;
  p.gm_plan = m.plan;
  p.tc_wait = c->tc_wait;
  p.err = &c->sc->err;
  return p;
}

IntParams int_params(md_ctx* c, double dt, const void* Br, const void* Bk) {
  IntParams p{};
  const md_config& g = c->cfg;
  const double a = c->alpha * c->L;
  p.n = (int)c->n;
  p.dt = dt;
  p.L = c->L;
  p.B_unit = B_unit(c);
  p.F_unit = F_unit(c);
  p.cself = 4.0 * a * a * a / (3.0 * std::sqrt(g.my_pi));
  p.csurf = 4.0 * g.my_pi / 3.0;
  p.anisConst = g.anisConst;
  p.velMmConst = g.velMmConst;
  p.magDamp = g.magDamp;
  p.mobil = (int)g.ENABLE_MOBILIZATION;
  p.noise = c->noise;
  p.seed = c->seed;
  p.field_kind = (int)g.fieldKind;
  p.magFluxDens = g.magFluxDens;
  p.tMag = g.tMag;
  p.fieldAmp = g.fieldAmp;
  p.fieldFreq = g.fieldFreq;
  p.xi = c->xi;
  p.pos = c->pos;
  p.mm = c->mm;
  p.ea = c->ea;
  p.truePos = c->truePos;
  p.posRef = c->posRef;
  p.magMom_u = c->magMom_u;
  p.rMag_u = c->rMag_u;
  p.cA = c->cA;
  p.cB = c->cB;
  p.f = IntParams::F32{(float)p.dt,     (float)p.L,     1.0f / (float)p.L,   (float)p.B_unit,     (float)p.F_unit,
                       (float)p.cself, (float)p.csurf, (float)p.anisConst, (float)p.velMmConst, (float)p.magDamp};
  p.k1m = c->k1m;
  p.k1e = c->k1e;
  p.m2 = c->m2;
  p.e2 = c->e2;
  p.th = c->th;
  p.Br = Br;
  p.Bk = Bk;
  p.Fr = c->Fr;
  p.Fk = c->Fk;
  p.ov = c->ov;
  p.mexact = nullptr;
  for (int q = 0; q < 6; q++) p.kself[q] = c->kself[q];
  p.sv = StrongView{};
  p.sv.flags = &c->sc->flags;
  if (strong_active(c)) {
    p.sv.off = c->snbr_off;
    p.sv.cap = c->scap;
    p.sv.B = Br == c->Br2 ? c->svals2 : c->svals;
    p.sv.F = c->svals + 3 * c->scap;
    p.sv.P = c->svals + 6 * c->scap;
  }
  p.s = sorted_view(c);
  p.musum = c->sc->musum;
  p.obs_part = c->obs_part;
  p.Ppart = c->Ppart;
  p.xbuild = c->xbuild;
  p.flags = &c->sc->flags;
  p.time = &c->sc->time;
  p.stepno = &c->sc->step;
  p.err = &c->sc->err;
  return p;
}

int check_ready(md_ctx* c, bool need_state) {
  if (!c) return set_err(nullptr, MD_ERR_INVALID, "null context");
  if (!c->have_particles) return set_err(c, MD_ERR_INVALID, "particles not set (md_set_particles)");
  if (!c->have_ewald) return set_err(c, MD_ERR_INVALID, "Ewald parameters not set (md_set_ewald)");
  if (need_state && !c->have_state) return set_err(c, MD_ERR_INVALID, "state not uploaded (md_state_upload)");
  return MD_OK;
}

// Real-space work and k-space work read the same sorted state and write
// separate outputs: they run concurrently, the k-space branch on the side
// stream (fork/join through events, which stream capture turns into parallel
// graph branches), so each fills the SMs the other's partial waves leave
// idle.  Each branch is a short preparation (neighbour list / phase tables)
// and its main kernels.  While per-segment profiling is on, everything runs
// on the main stream in the order prep, prep, real, k-space, with the
// segment events before the real and the k-space kernels.
template <class RP, class RM, class KP, class KM>
static int fork_join(md_ctx* c, int q, int seg_real, int seg_k, RP&& real_prep, RM&& real, KP&& k_prep,
                     KM&& kspace) {
  if (c->prof) {
    int l = real_prep(c->stream) + k_prep(c->stream);
    mark(c, seg_real);
    l += real(c->stream);
    mark(c, seg_k);
    return l + kspace(c->stream);
  }
  cudaEventRecord(c->fork_ev[q], c->stream);
  cudaStreamWaitEvent(c->side, c->fork_ev[q], 0);
  int l = k_prep(c->side) + kspace(c->side);
  l += real_prep(c->stream) + real(c->stream);
  cudaEventRecord(c->join_ev[q], c->side);
  cudaStreamWaitEvent(c->stream, c->join_ev[q], 0);
  return l;
}

// Field + force evaluation on the current master state (no integrator).
// dt >= 0: the step's noise is drawn beside it (unit: see launch_noise).  after_records: the step before left
// its records to the side stream (issue_step); they come before the noise, and with
// it the integrator.
static int issue_interactions(md_ctx* c, double dt = -1.0, bool unit = false, bool after_records = false) {
  int l = 0;
  mark(c, MD_SEG_CELLS);
  if (!c->list_valid) c->cell_skin = c->skin_frac;  // this evaluation sorts anew
  const CellParams cp = cell_params(c);
  const KParams kp = k_params(c, nullptr, nullptr);
  const bool fused = fill_phases_fused(kp);
  l += launch_cells(c->stream, cp, fp64(c), !fused);
  if (fused) l += launch_fill_phases(c->stream, cp, kp, fp64(c));
  l += fork_join(
      c, 0, MD_SEG_REAL_FULL, MD_SEG_KSF_FULL,
      [&](cudaStream_t st) {
        int l = launch_nbr(st, real_params(c, nullptr, nullptr, nullptr), fp64(c));
        if (after_records) cudaStreamWaitEvent(st, c->join_ev[2], 0);
        if (dt >= 0) l += launch_noise(st, int_params(c, dt, nullptr, nullptr), unit, fp64(c));
        return l;
      },
      [&](cudaStream_t st) { return launch_real(st, real_params(c, c->Br, c->Fr, c->ov), true, fp64(c)); },
      [&](cudaStream_t st) { return fused ? 0 : launch_phase_tables(st, kp); },
      [&](cudaStream_t st) {
        return launch_kspace(st, k_params(c, c->Bk, c->Fk), true, fp64(c),
                             c->prof ? &c->ev[MD_SEG_KRED_FULL] : nullptr);
      });
  c->have_geometry = true;
  c->list_valid = true;
  return l;
}

// Field-only evaluation (CompDemagField) for the moments in the sorted view.
static int issue_field(md_ctx* c) {
  auto none = [](cudaStream_t) { return 0; };
  return fork_join(
      c, 1, MD_SEG_REAL_FIELD, MD_SEG_KSF_FIELD, none,
      [&](cudaStream_t st) { return launch_real(st, real_params(c, c->Br2, nullptr, nullptr), false, fp64(c)); },
      none,
      [&](cudaStream_t st) {
        return launch_kspace(st, k_params(c, c->Bk2, nullptr), false, fp64(c),
                             c->prof ? &c->ev[MD_SEG_KRED_FIELD] : nullptr);
      });
}

// leave_records: another step follows in the same graph, and the records of this
// one are taken beside the start of that one (the kernel that ends with them in its
// last block costs the chain of steps ~2 us more: N = 512 49.0 -> 46.8 us per step).
static int issue_step(md_ctx* c, double dt, bool after_records = false, bool leave_records = false) {
  int l = issue_interactions(c, dt, false, after_records);
  mark(c, MD_SEG_HEUN1);
  l += launch_heun1(c->stream, int_params(c, dt, c->Br, c->Bk), fp64(c));
  l += issue_field(c);
  mark(c, MD_SEG_HEUN2);
  const IntParams ip = int_params(c, dt, c->Br2, c->Bk2);
  const ObsParams op = obs_params(c, dt);
  if (leave_records) {
    l += launch_heun2(c->stream, ip, fp64(c));
    cudaEventRecord(c->fork_ev[2], c->stream);
    cudaStreamWaitEvent(c->side, c->fork_ev[2], 0);
    l += launch_records(c->side, op, (int)c->n);
    cudaEventRecord(c->join_ev[2], c->side);
    return l;
  }
  l += launch_heun2_obs(c->stream, ip, op, &c->sc->done, fp64(c));
  mark(c, MD_SEG_OBS);  // the records are taken inside the stage-2 launch
  mark(c, MD_NSEG);
  return l;
}

// In-range pairs of the last evaluation, counted while its list is still there
// (before new particles, box, cut-off or skin) and on request.
static int count_pairs(md_ctx* c) {
  if (!c->list_valid) return MD_OK;
  unsigned long long v = 0;
  CK(c, cudaMemsetAsync(&c->sc->pairs, 0, sizeof v, c->stream));
  launch_count_pairs(c->stream, real_params(c, nullptr, nullptr, nullptr), &c->sc->pairs, fp64(c));
  CK(c, cudaMemcpyAsync(&v, &c->sc->pairs, sizeof v, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  c->pairs = (int64_t)(v / 2);
  return MD_OK;
}

// Asks the device to rebuild the cell order and the neighbour list at the
// start of the next evaluation.
int force_rebuild(md_ctx* c) {
  static const int one = 1;
  CK(c, cudaMemcpyAsync(&c->sc->flags.force, &one, sizeof(int), cudaMemcpyHostToDevice, c->stream));
  return MD_OK;
}

// Capacity of the neighbour list.  keep: the current list stays (field evaluations
// at the last geometry still read it), unless there is no memory for both.
int alloc_nbr(md_ctx* c, long long cap, bool keep) {
  cap = std::min<long long>(cap, 0x7ffffffeLL);
  if (cap <= c->nbr_cap) return MD_OK;
  int* list = nullptr;
  if (keep && c->have_geometry && c->nbr) {
    const size_t at = (size_t)(std::find(c->allocs.begin(), c->allocs.end(), (void*)c->nbr) - c->allocs.begin());
    const size_t held = std::min(c->alloc_bytes[at], 4 * (size_t)cap);
    if (dalloc(c, &list, 4 * (size_t)cap) == MD_OK) {
      CK(c, cudaMemcpyAsync(list, c->nbr, held, cudaMemcpyDeviceToDevice, c->stream));
    } else {
      cudaGetLastError();
      c->have_geometry = false;
    }
  }
  dfree(c, c->nbr);
  c->nbr = list;
  c->nbr_cap = 0;
  if (!list)
    if (int st = dalloc(c, &c->nbr, 4 * (size_t)cap)) return st;
  c->nbr_cap = cap;
  invalidate_graph(c);
  return MD_OK;
}

bool strong_active(const md_ctx* c) {
  return !fp64(c) && !c->cfg.ENABLE_COATING_POT && c->strong_w4sq > 0.f && c->scap > 0 && c->snbr_off;
}

int alloc_strong(md_ctx* c, long long cap) {
  cap = std::min<long long>(cap, 0x7ffffffeLL);
  if (cap <= c->scap) return MD_OK;
  dfree(c, c->snbr);
  dfree(c, c->svals);
  dfree(c, c->svals2);
  c->snbr = nullptr;
  c->svals = c->svals2 = nullptr;
  c->scap = 0;
  int st = dalloc(c, &c->snbr, sizeof(int2) * (size_t)cap);
  if (!st) st = dalloc(c, &c->svals, 9 * sizeof(double) * (size_t)cap);
  if (!st) st = dalloc(c, &c->svals2, 3 * sizeof(double) * (size_t)cap);
  if (st) return st;
  c->scap = cap;
  invalidate_graph(c);
  // not in use before the next build has filled it (a field at the last geometry
  // takes every pair in FP32)
  static const int one = 1;
  CK(c, cudaMemcpyAsync(&c->sc->flags.soverflow, &one, sizeof(int), cudaMemcpyHostToDevice, c->stream));
  return MD_OK;
}

// Threshold of the strong pairs in kernel units: the force weight
// (|mu_i| |mu_j| / mu_min^2) (d_min / r)^4, d_min = 2 min rHydr (the scale
// of the reference's relative error, src/interaction.cpp:180), exceeds
// strong_theta  <=>  |mu_i|^2 |mu_j|^2 > w4sq r^8 with moments in mu_max
// and r in box lengths.  A monodisperse system has no pair above theta >= 1.
void update_strong(md_ctx* c) {
  c->strong_w4sq = -1.f;
  if (fp64(c) || !(c->strong_theta > 0) || !c->have_particles || c->props.magMom.empty()) return;
  double mmin = 1e300, rhmin = 1e300;
  for (size_t i = 0; i < c->props.magMom.size(); i++) {
    mmin = std::min(mmin, c->props.magMom[i]);
    rhmin = std::min(rhmin, c->props.rHydr[i]);
  }
  const double q = mmin / c->props.muMax, dl = c->L / (2.0 * rhmin);
  const double w4 = c->strong_theta * q * q * dl * dl * dl * dl;
  const double w4sq = w4 * w4;
  c->strong_w4sq = w4sq < 3.0e38 ? (float)w4sq : -1.f;
}

// Expected entries of the strong list at uniform density: particles binned
// by log moment (48 bins; per bin the largest moment and the smallest
// hydrodynamic radius, so the estimate errs high), and per bin pair the
// shell between contact and the distance where the weight falls to theta
// (2 * 1.25e5 entries estimated vs 1.22e5 built for N = 32768, log-normal
// sigma 0.2).
static double strong_estimate(const mdh::Props& p, double L, double rl, double theta) {
  const std::vector<double>& m = p.magMom;
  const std::vector<double>& rh = p.rHydr;
  if (m.empty() || !(theta > 0)) return 0;
  double mmin = 1e300, mmax = 0, rhmin = 1e300;
  for (size_t i = 0; i < m.size(); i++) {
    mmin = std::min(mmin, m[i]);
    mmax = std::max(mmax, m[i]);
    rhmin = std::min(rhmin, rh[i]);
  }
  const int nb = 48;
  const double span = std::log(mmax / mmin) * (1.0 + 1e-9) + 1e-12;
  std::vector<double> cnt(nb, 0.0), mb(nb, 0.0), rb(nb, 1e300);
  for (size_t i = 0; i < m.size(); i++) {
    const int b = std::min(nb - 1, (int)(std::log(m[i] / mmin) / span * nb));
    cnt[b] += 1;
    mb[b] = std::max(mb[b], m[i]);
    rb[b] = std::min(rb[b], rh[i]);
  }
  const double pi = 3.141592653589793, V = L * L * L, dmin = 2.0 * rhmin;
  double tot = 0;
  for (int a = 0; a < nb; a++)
    for (int b = 0; b < nb; b++) {
      if (cnt[a] == 0 || cnt[b] == 0) continue;
      const double rs = dmin * std::pow(mb[a] * mb[b] / (mmin * mmin * theta), 0.25);
      const double rc = std::min(rs, rl), cont = rb[a] + rb[b];
      if (rc > cont) tot += cnt[a] * cnt[b] * 4.0 / 3.0 * pi * (rc * rc * rc - cont * cont * cont) / V;
    }
  return tot;
}

static long long strong_entries(const md_ctx* c) {
  return 4096 + (long long)(2.0 * strong_estimate(c->props, c->L, c->rc * (1.0 + c->skin_frac), c->strong_theta));
}

// After work on the stream: a neighbour list that did not fit was replaced by
// the direct cell scan (results are correct); grow it for the next steps.
static int handle_overflow(md_ctx* c, const StepFlags& f);

int check_overflow(md_ctx* c) {
  StepFlags f;
  CK(c, cudaMemcpyAsync(&f, &c->sc->flags, sizeof f, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return handle_overflow(c, f);
}

static int handle_overflow(md_ctx* c, const StepFlags& f) {
  if (f.soverflow && !f.overflow && strong_active(c)) {
    // the strong list did not fit (or the last build did not classify):
    // grow it if needed and classify again at the next step
    int total = 0;
    CK(c, cudaMemcpy(&total, c->snbr_off + c->n, sizeof(int), cudaMemcpyDeviceToHost));
    if (total > c->scap || total < 0) {
      const long long need = (total > 0 && total < 0x7fffffff) ? (long long)(total * 1.25) + 4LL * c->n : 2 * c->scap;
      if (int st = alloc_strong(c, need)) return st;
    }
    if (int st = force_rebuild(c)) return st;
  }
  if (!f.overflow) return MD_OK;
  int total = 0;
  CK(c, cudaMemcpy(&total, c->nbr_off + c->n, sizeof(int), cudaMemcpyDeviceToHost));
  const long long need = (total > 0 && total < 0x7fffffff) ? (long long)(total * 1.25) + 16LL * c->n : 2 * c->nbr_cap;
  int st = alloc_nbr(c, need);
  if (st) return st;
  // The overflow flag stays set until the next rebuild (which recounts the
  // list against the new capacity): a field-only evaluation before that
  // (md_compute_field) must scan the cells, since the list was never filled.
  return force_rebuild(c);
}

// Error word and list flags of the work on the stream, read together (one
// copy of the device scalars, one synchronisation).
int read_err_word(md_ctx* c) {
  DevScalars h;
  CK(c, cudaMemcpyAsync(&h, c->sc, sizeof h, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  const int e = h.err;
  if (e) {
    CK(c, cudaMemsetAsync(&c->sc->err, 0, sizeof(int), c->stream));
    if (e & kErrNonFinite) return set_err(c, MD_ERR_NONFINITE, "non-finite position or orientation after the step");
    if (e & kErrTcWait) return set_err(c, MD_ERR_CUDA, "tensor-core k space: a pipeline wait gave up");
  }
  return handle_overflow(c, h.flags);
}

// ============================================================== C ABI

// Largest kc the context's k space runs on the tensor cores (0: none).
static int tc_kc_bound(const md_ctx* c) {
  return (fp64(c) || c->kengine == MD_KSPACE_SIMT) ? 0 : md::kspace_tc_max_kc();
}

static int num_sms(int device) {
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  return nsm;
}

// Cells: a stencil of +-2 on the FP64 path; on the mixed path ~4 particles
// each, which keeps the two consecutive sorted particles whose lists one
// warp builds close together and fits the cells to the search sphere.
static CellGrid cell_grid(double rc_box, int64_t n, bool f64) {
  const int reach = f64 ? 2 : (int)std::lround(rc_box * std::cbrt(0.25 * (double)n));
  return mdh::choose_grid(rc_box, n, std::max(2, std::min(reach, 12)));
}

// Structure-factor grid of the row segments (segment blocks x particle chunks): the
// fewest whole waves of resident blocks that keep every FP32 chunk sum within 512
// particles, with the chunk count chosen to fill those waves.
static void segment_chunks(const mdh::KList& k, int64_t n, int kc, int nsm, int* chunk, int* nchunk) {
  const int nsegb = (int)((k.seg.size() + md::sk_threads() - 1) / md::sk_threads());
  const int64_t slots = (int64_t)nsm * md::sk_resident_blocks(kc);
  const int64_t nch_min = std::max<int64_t>(1, (n + 511) / 512);
  const int64_t waves = std::max<int64_t>(1, (nsegb * nch_min + slots - 1) / slots);
  int64_t nch = std::max<int64_t>(nch_min, waves * slots / nsegb);
  nch = std::min<int64_t>(nch, (n + 31) / 32);
  *chunk = (int)(((n + nch - 1) / nch + 31) / 32 * 32);
  *nchunk = (int)((n + *chunk - 1) / *chunk);
}

void ctx_packed_only(md_ctx* c) { c->packed_only = true; }

// Tensor-core k space: the k rows (ny, nz) of the half-space k list, ordered
// by nz then ny, the k index of each (row, nx), and the buffers of the
// launches (md_ktc.cu).  Off (tc_rows = 0) on the FP64 path, when the
// engine is MD_KSPACE_SIMT, or when kc is beyond the kernels' shared memory.
static int setup_tc(md_ctx* c) {
  c->tc_rows = 0;
  if (fp64(c) || c->kengine == MD_KSPACE_SIMT || !md::kspace_tc_supported((int)c->kc)) return MD_OK;
  const int kc = (int)c->kc, Q = 2 * kc + 1, nk = c->klist.nk;
  std::map<std::pair<int, int>, int> rowid;  // (nz, ny) -> row
  for (int k = 0; k < nk; k++)
    if (c->klist.kreal[k]) rowid[{c->klist.kz[k], c->klist.ky[k]}] = 0;
  std::vector<int2> rows;
  for (auto& e : rowid) {
    e.second = (int)rows.size();
    rows.push_back(make_int2(e.first.second, e.first.first));
  }
  const int R = (int)rows.size();
  if (R == 0) return MD_OK;
  std::vector<int> kmap((size_t)R * Q, -1);
  for (int k = 0; k < nk; k++)
    if (c->klist.kreal[k]) kmap[(size_t)rowid[{c->klist.kz[k], c->klist.ky[k]}] * Q + c->klist.kx[k] + kc] = k;
  const md::TcShape t = md::kspace_tc_shape(kc, (int)c->n, R, num_sms(c->device), c->tc_ring, c->tc_waves);
  void* old[] = {c->tc_row, c->tc_rowd, c->tc_kmap, c->tc_part, c->tc_wfull, c->tc_wfield, c->tc_bimg, c->tc_tblk};
  for (void* q : old) dfree(c, q);
  c->tc_row = nullptr;
  c->tc_rowd = nullptr;
  c->tc_kmap = nullptr;
  c->tc_part = nullptr;
  c->tc_wfull = c->tc_wfield = nullptr;
  c->tc_bimg = nullptr;
  c->tc_tblk = nullptr;
  const size_t wfull = md::kspace_tc_image_floats(kc, t.nt_full), wfield = md::kspace_tc_image_floats(kc, t.nt_field);
  int st;
  if ((st = dalloc(c, &c->tc_row, sizeof(int2) * (size_t)R))) return st;
  std::vector<float4> rowd((size_t)md::kspace_tc_rows_pad(R));
  md::kspace_tc_row_desc(rows.data(), R, kc, (int)c->n, t.yz != 0, rowd.data());
  if ((st = dalloc(c, &c->tc_rowd, sizeof(float4) * rowd.size()))) return st;
  if ((st = dalloc(c, &c->tc_kmap, sizeof(int) * kmap.size()))) return st;
  if ((st = dalloc(c, &c->tc_part, sizeof(float) * (size_t)t.nchunk * t.mt * t.ns * 128))) return st;
  if ((st = dalloc(c, &c->tc_wfull, sizeof(float) * wfull))) return st;
  if ((st = dalloc(c, &c->tc_wfield, sizeof(float) * wfield))) return st;
  if ((st = dalloc(c, &c->tc_bimg, sizeof(float) * md::kspace_tc_bimg_floats(kc, t.nsb)))) return st;
  if ((st = dalloc(c, &c->tc_tblk, sizeof(float2) * md::kspace_tc_tblk_entries(kc, t.nsb)))) return st;
  if (t.nchunk > c->musum_cap) {
    dfree(c, c->musum_part);
    c->musum_part = nullptr;
    if ((st = dalloc(c, &c->musum_part, 24 * (size_t)t.nchunk))) return st;
    c->musum_cap = t.nchunk;
  }
  CK(c, cudaMemcpy(c->tc_row, rows.data(), sizeof(int2) * (size_t)R, cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->tc_rowd, rowd.data(), sizeof(float4) * rowd.size(), cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->tc_kmap, kmap.data(), sizeof(int) * kmap.size(), cudaMemcpyHostToDevice));
  // operand entries of k's outside the sphere or the half space stay zero
  CK(c, cudaMemset(c->tc_wfull, 0, sizeof(float) * wfull));
  CK(c, cudaMemset(c->tc_wfield, 0, sizeof(float) * wfield));
  c->tcs = t;
  c->tc_rows = R;
  return MD_OK;
}

// Whether the mixed path's default engine takes the row kernels (md_krows.cu)
// instead of the tensor cores: systems of up to 3e6 (k, particle) terms, whose
// tensor-core launches are mostly set-up.  Measured step times, rows against
// tensor cores: N = 512, kc = 7 (0.4e6 terms) 66 / 84 us, N = 1000, kc = 7 (0.7e6)
// 80 / 86, N = 2048, kc = 8 (2.2e6) 90 / 94; N = 4096, kc = 9 (6.3e6) 120 / 105,
// N = 3001, kc = 11 (8.4e6) 130 / 119.  An engine or a tensor-core tiling that
// the caller chose is kept.
static bool krows_wanted(const md_ctx* c) {
  const double nk = 2.0943951 * (double)c->kc * (double)c->kc * (double)c->kc;  // half space
  return c->kengine == MD_KSPACE_AUTO && !c->packed_only && c->tc_ring < 0 && c->tc_waves == 1 &&
         md::kspace_tc_supported((int)c->kc) && nk * (double)c->n <= 3e6;
}

// k space by rows: tasks of four consecutive |nx| of one k row, rows by nz
// then ny, and the buffers of the launches (md_krows.cu).  Always on the FP64
// path, on the mixed path for the systems of krows_wanted.
static int setup_rows(md_ctx* c) {
  c->rw_T = c->rw_R = 0;
  if (!fp64(c) && !krows_wanted(c)) return MD_OK;
  const int kc = (int)c->kc, nk = c->klist.nk;
  std::map<std::pair<int, int>, std::vector<std::pair<int, int>>> byrow;  // (nz, ny) -> (nx, k)
  for (int k = 0; k < nk; k++)
    if (c->klist.kreal[k]) byrow[{c->klist.kz[k], c->klist.ky[k]}].push_back({c->klist.kx[k], k});
  std::vector<int4> task;
  std::vector<int> kidx;
  std::vector<double2> row;
  std::vector<int2> rowt;
  for (const auto& e : byrow) {
    const int nz = e.first.first, ny = e.first.second;
    int top = 0;
    for (const auto& q : e.second) top = std::max(top, std::abs(q.first));
    const int nt = top / 4 + 1, t0 = (int)task.size();
    for (int t = 0; t < nt; t++) task.push_back(make_int4((int)row.size(), ny, nz, 4 * t));
    kidx.resize(8 * task.size(), -1);
    for (const auto& q : e.second) {
      const int ax = std::abs(q.first);
      kidx[8 * (size_t)(t0 + ax / 4) + 2 * (ax % 4) + (q.first < 0 ? 1 : 0)] = q.second;
    }
    row.push_back(make_double2((double)ny, (double)nz));
    rowt.push_back(make_int2(t0, nt));
  }
  const int T = (int)task.size(), R = (int)row.size();
  const md::RowShape sh = md::krows_shape(kc, (int)c->n, T, num_sms(c->device), fp64(c));
  void* old[] = {c->rw_task, c->rw_kidx, c->rw_row, c->rw_rowt, c->rw_ad};
  for (void* q : old) dfree(c, q);
  c->rw_task = nullptr;
  c->rw_kidx = nullptr;
  c->rw_row = nullptr;
  c->rw_rowt = nullptr;
  c->rw_ad = nullptr;
  int st;
  if ((st = dalloc(c, &c->rw_task, sizeof(int4) * (size_t)T))) return st;
  if ((st = dalloc(c, &c->rw_kidx, sizeof(int) * kidx.size()))) return st;
  if ((st = dalloc(c, &c->rw_row, sizeof(double2) * (size_t)R))) return st;
  if ((st = dalloc(c, &c->rw_rowt, sizeof(int2) * (size_t)R))) return st;
  if ((st = dalloc(c, &c->rw_ad, 16 * tsz(c) * (size_t)T))) return st;
  const size_t sp = tsz(c) * (size_t)T * (size_t)sh.nchunk;  // 16 T per task and chunk, in double2
  if (sp > c->spart_cap) {
    dfree(c, c->Spart);
    c->Spart = nullptr;
    c->spart_cap = 0;
    if ((st = dalloc(c, &c->Spart, sizeof(double2) * sp))) return st;
    c->spart_cap = sp;
  }
  if (sh.nchunk > c->musum_cap) {
    dfree(c, c->musum_part);
    c->musum_part = nullptr;
    c->musum_cap = 0;
    if ((st = dalloc(c, &c->musum_part, 24 * (size_t)sh.nchunk))) return st;
    c->musum_cap = sh.nchunk;
  }
  CK(c, cudaMemcpy(c->rw_task, task.data(), sizeof(int4) * (size_t)T, cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->rw_kidx, kidx.data(), sizeof(int) * kidx.size(), cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->rw_row, row.data(), sizeof(double2) * (size_t)R, cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->rw_rowt, rowt.data(), sizeof(int2) * (size_t)R, cudaMemcpyHostToDevice));
  c->rws = sh;
  c->rw_T = T;
  c->rw_R = R;
  return MD_OK;
}

// Whether the mixed path's default engine goes through a mesh (md_kmesh.cu)
// instead of the tensor cores.  The mesh's work is in its particles and, ~M^3, in its
// transforms, the tensor cores' in particles x k vectors, in steps (at kc = 20 and 24
// they pad most).  Step times, mesh against tensor cores, both splits from the error
// model:
//   N = 20011 and more   10 to 37 % shorter (kc = 15 .. 25)
//   N = 14000 .. 16384   up to 17 % shorter, 5 % longer at worst (kc = 17); kc = 25
//                        (M^3 = 80 N) 3 % longer at 14000, 4 % shorter at 15000
//   N = 8192 .. 13000    kc = 20 5 to 10 %, kc = 24 2 to 9 % shorter, kc = 16 equal to 6 %
//                        shorter; the others 2 to 16 % longer
//   N = 6000             2 to 18 % longer
//   N = 32768, kc = 13   621 / 626 us, kc = 12 609 / 595
// Where it takes longer it stays for its error, an eighth of the tensor cores' in the
// field (k-space part against FP64, rms, N = 32768: field 1.5e-7 / 1.2e-6, force 2.8e-7
// / 1.3e-6); from M^3 = 100 N on and below 6000 particles the time decides.  An engine
// or a tensor-core tiling that the caller chose is kept.
static bool mesh_wanted(const md_ctx* c) {
  if (fp64(c) || c->kengine != MD_KSPACE_AUTO || c->packed_only || c->tc_ring >= 0 || c->tc_waves != 1 || c->tc_rows == 0) return false;
  const double M = md::mesh_points((int)c->kc);
  return c->n >= 6000 && (c->kc >= 15 || (c->kc >= 13 && c->n >= 32768)) && M * M * M <= 100.0 * (double)c->n;
}

// k space through a mesh: window tables and the mesh in its stages (md_kmesh.cu).
static int setup_mesh(md_ctx* c) {
  c->gm_M = 0;
  if (!mesh_wanted(c)) return MD_OK;
  const int kc = (int)c->kc, M = md::mesh_points(kc), items = md::mesh_items(M);
  const size_t kc1 = (size_t)kc + 1, rows = kc1 * (2 * (size_t)kc + 1), M2 = (size_t)M * M;
  const mdh::MeshTables t = mdh::mesh_tables(kc, M);
  // factors in the layout of tc_kmap: row, nx
  const int Q = 2 * kc + 1;
  std::map<std::pair<int, int>, int> rowid;
  for (int k = 0; k < c->klist.nk; k++)
    if (c->klist.kreal[k]) rowid[{c->klist.kz[k], c->klist.ky[k]}] = 0;
  int nr = 0;
  for (auto& e : rowid) e.second = nr++;
  std::vector<float2> fac((size_t)nr * Q, make_float2(0.f, 0.f));
  for (int k = 0; k < c->klist.nk; k++)
    if (c->klist.kreal[k]) {
      const int nx = c->klist.kx[k], ny = c->klist.ky[k], nz = c->klist.kz[k];
      const double d = t.dec[std::abs(nx)] * t.dec[std::abs(ny)] * t.dec[nz];
      fac[(size_t)rowid[{nz, ny}] * Q + nx + kc] = make_float2((float)(c->klist.ek[k] * d * d), (float)d);
    }
  std::vector<float2> tw(M);
  for (int j = 0; j < M; j++) {
    const double a = 2.0 * std::acos(-1.0) * j / M;
    tw[j] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  void* old[] = {c->gm_coef, c->gm_fac, c->gm_tw, c->gm_part, c->gm_z, c->gm_y, c->gm_t, c->gm_b, c->gm_plan};
  for (void* q : old) dfree(c, q);
  c->gm_coef = nullptr;
  c->gm_fac = nullptr;
  c->gm_tw = nullptr;
  c->gm_part = nullptr;
  c->gm_z = nullptr;
  c->gm_y = c->gm_t = c->gm_b = nullptr;
  c->gm_plan = nullptr;
  std::vector<int> plan;
  md::mesh_plan_init(M, plan);
  int st;
  if ((st = dalloc(c, &c->gm_coef, sizeof(float) * t.coef.size()))) return st;
  if ((st = dalloc(c, &c->gm_fac, sizeof(float2) * fac.size()))) return st;
  if ((st = dalloc(c, &c->gm_tw, sizeof(float2) * (size_t)M))) return st;
  if ((st = dalloc(c, &c->gm_part, sizeof(float) * md::mesh_part_floats(M)))) return st;
  if ((st = dalloc(c, &c->gm_z, sizeof(float2) * 3 * kc1 * M2))) return st;
  if ((st = dalloc(c, &c->gm_y, sizeof(float4) * rows * M))) return st;
  if ((st = dalloc(c, &c->gm_t, sizeof(float4) * rows * M))) return st;
  if ((st = dalloc(c, &c->gm_b, sizeof(float4) * M2 * M))) return st;
  if ((st = dalloc(c, &c->gm_plan, sizeof(int) * plan.size()))) return st;
  if (items > c->musum_cap) {
    dfree(c, c->musum_part);
    c->musum_part = nullptr;
    c->musum_cap = 0;
    if ((st = dalloc(c, &c->musum_part, 24 * (size_t)items))) return st;
    c->musum_cap = items;
  }
  CK(c, cudaMemcpy(c->gm_coef, t.coef.data(), sizeof(float) * t.coef.size(), cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->gm_fac, fac.data(), sizeof(float2) * fac.size(), cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->gm_tw, tw.data(), sizeof(float2) * (size_t)M, cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->gm_plan, plan.data(), sizeof(int) * plan.size(), cudaMemcpyHostToDevice));
  c->gm_M = M;
  return MD_OK;
}

// The k-space engine of the current parameters.
static int setup_engine(md_ctx* c) {
  int st = setup_tc(c);
  if (!st) st = setup_rows(c);
  return st ? st : setup_mesh(c);
}

extern "C" {

const char* md_strerror(int s) {
  switch (s) {
    case MD_OK: return "ok";
    case MD_ERR_INVALID: return "invalid argument or state";
    case MD_ERR_CUDA: return "CUDA runtime error";
    case MD_ERR_NOMEM: return "out of memory";
    case MD_ERR_NONFINITE: return "non-finite value in the simulation state";
    case MD_ERR_CONFIG: return "configuration error";
    case MD_ERR_UNSUPPORTED: return "unsupported";
    case MD_ERR_NO_DEVICE: return "no CUDA device";
    default: return "unknown status";
  }
}

int md_last_error(const md_ctx* c, char* buf, size_t len) {
  std::string m;
  int st;
  if (c) {
    m = c->err;
    st = c->err_status;
  } else {
    std::lock_guard<std::mutex> lk(g_err_mu);
    m = g_err;
    st = g_err_status;
  }
  if (buf && len) {
    std::strncpy(buf, m.c_str(), len - 1);
    buf[len - 1] = 0;
  }
  return st;
}

const char* md_version(void) { return "md_gb300 1.0 (sm_103a)"; }

int md_config_default(md_config* cfg) {
  if (!cfg) return set_err(nullptr, MD_ERR_INVALID, "null config");
  mdh::config_defaults(cfg);
  return MD_OK;
}

int md_config_derive(md_config* cfg) {
  if (!cfg) return set_err(nullptr, MD_ERR_INVALID, "null config");
  mdh::config_derive(cfg);
  return MD_OK;
}

int md_config_load_ini(const char* path, md_config* cfg) {
  if (!path || !cfg) return set_err(nullptr, MD_ERR_INVALID, "null argument");
  std::string e;
  int st = mdh::config_load_ini(path, cfg, &e);
  if (st) return set_err(nullptr, st, "%s", e.c_str());
  return MD_OK;
}

int64_t md_config_numb_part(const md_config* cfg) { return cfg ? mdh::numb_part(cfg) : 0; }

size_t md_config_size(void) { return sizeof(md_config); }

int md_select_device(int device) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_err(nullptr, MD_ERR_NO_DEVICE, "cudaSetDevice(%d): %s", device, cudaGetErrorString(e));
  }
  return MD_OK;
}

int md_ctx_create(const md_config* cfg, int64_t n, int precision, md_ctx** out) {
  if (!cfg || !out || n < 2 || n > (1LL << 30)) return set_err(nullptr, MD_ERR_INVALID, "bad md_ctx_create arguments");
  if (precision != MD_PREC_FP64 && precision != MD_PREC_MIXED)
    return set_err(nullptr, MD_ERR_INVALID, "unknown precision %d", precision);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return set_err(nullptr, MD_ERR_NO_DEVICE, "no CUDA device visible");
  }
  md_ctx* c = new md_ctx();
  c->cfg = *cfg;
  c->n = n;
  c->prec = precision;
  c->noise = (int)cfg->noise;
  c->seed = (uint64_t)cfg->seed;
  cudaGetDevice(&c->device);
  int st = MD_OK;
  auto fail = [&](int s) {
    md_ctx_destroy(c);
    return s;
  };
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking) != cudaSuccess)
    return fail(set_err(nullptr, MD_ERR_CUDA, "cudaStreamCreate failed"));
  pool_keep(c->device);
  for (int q = 0; q < 3; q++)
    if (cudaEventCreateWithFlags(&c->fork_ev[q], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->join_ev[q], cudaEventDisableTiming) != cudaSuccess)
      return fail(set_err(nullptr, MD_ERR_CUDA, "cudaEventCreate failed"));
  const size_t N = (size_t)n, T = tsz(c);
  double** d3[] = {&c->pos, &c->mm, &c->ea, &c->truePos, &c->posRef, &c->tmpmm, &c->Bout, &c->Fout};
  for (auto p : d3)
    if ((st = dalloc(c, p, 24 * N))) return fail(st);
  if ((st = dalloc(c, &c->xi, 72 * N))) return fail(st);
  double** d1[] = {&c->magMom_u, &c->rMag_u, &c->invZt, &c->velEa1, &c->velEa2, &c->zetaR, &c->zetaT, &c->invVol};
  for (auto p : d1)
    if ((st = dalloc(c, p, 8 * N))) return fail(st);
  int** i1[] = {&c->cellOf, &c->tmp, &c->perm, &c->rank, &c->scell};
  for (auto p : i1)
    if ((st = dalloc(c, p, 4 * N))) return fail(st);
  if ((st = dalloc(c, &c->xf, 16 * N))) return fail(st);
  if (fp64(c)) {
    if ((st = dalloc(c, &c->xd, 32 * N))) return fail(st);
  } else {
    if ((st = dalloc(c, &c->xi4, 16 * N))) return fail(st);
  }
  if ((st = dalloc(c, &c->mu, 4 * T * N))) return fail(st);
  if ((st = dalloc(c, &c->cA, 4 * T * N)) || (st = dalloc(c, &c->cB, 4 * T * N)) ||
      (st = dalloc(c, &c->sTB, 16 * N)))
    return fail(st);
  void** t3[] = {&c->Br, &c->Fr, &c->ov, &c->Bk, &c->Fk, &c->Br2, &c->Bk2, &c->k1m, &c->k1e, &c->m2, &c->e2};
  for (auto p : t3)
    if ((st = dalloc(c, p, 3 * T * N))) return fail(st);
  if ((st = dalloc(c, &c->th, 9 * T * N))) return fail(st);
  if ((st = dalloc(c, &c->nbr_cnt, 4 * N))) return fail(st);
  if ((st = dalloc(c, &c->nbr_off, 4 * (N + 1)))) return fail(st);
  if ((st = dalloc(c, &c->xbuild, 24 * N))) return fail(st);
  if ((st = dalloc(c, &c->Ppart, 24 * N))) return fail(st);
  if ((st = dalloc(c, &c->obs_part, 56 * (size_t)std::max(int_blocks((int)n), int_blocks_one((int)n))))) return fail(st);
  if (!fp64(c)) {
    if ((st = dalloc(c, &c->snbr_cnt, 4 * N)) || (st = dalloc(c, &c->snbr_off, 4 * (N + 1)))) return fail(st);
    if (cudaMemsetAsync(c->snbr_off, 0, 4 * (N + 1), c->stream) != cudaSuccess)
      return fail(set_err(nullptr, MD_ERR_CUDA, "initial memset failed"));
  }
  if ((st = dalloc(c, &c->sc, sizeof(DevScalars)))) return fail(st);
  if (fp64(c)) {
    const mdh::RealTables t = mdh::real_tables64(cfg->irPi);
    if ((st = dalloc(c, &c->gtab, 8 * t.g.size())) || (st = dalloc(c, &c->etab, 8 * t.e.size()))) return fail(st);
    if (cudaMemcpyAsync(c->gtab, t.g.data(), 8 * t.g.size(), cudaMemcpyHostToDevice, c->stream) != cudaSuccess ||
        cudaMemcpyAsync(c->etab, t.e.data(), 8 * t.e.size(), cudaMemcpyHostToDevice, c->stream) != cudaSuccess ||
        cudaStreamSynchronize(c->stream) != cudaSuccess)
      return fail(set_err(nullptr, MD_ERR_CUDA, "table upload failed"));
  }
  static const int one = 1;
  if (cudaMemsetAsync(c->sc, 0, sizeof(DevScalars), c->stream) != cudaSuccess ||
      cudaMemcpyAsync(&c->sc->flags.soverflow, &one, sizeof(int), cudaMemcpyHostToDevice, c->stream) != cudaSuccess ||
      cudaMemsetAsync(c->xi, 0, 72 * N, c->stream) != cudaSuccess ||
      cudaMemsetAsync(c->Ppart, 0, 24 * N, c->stream) != cudaSuccess)
    return fail(set_err(nullptr, MD_ERR_CUDA, "initial memset failed"));
  *out = c;
  return MD_OK;
}

int md_ctx_destroy(md_ctx* c) {
  if (!c) return MD_OK;
  if (c->stream) cudaStreamSynchronize(c->stream);
  invalidate_graph(c);
  for (auto& e : c->ev)
    if (e) cudaEventDestroy(e);
  if (c->side) cudaStreamSynchronize(c->side);
  for (void* p : c->allocs) cudaFreeAsync(p, c->stream);
  if (c->stream) cudaStreamSynchronize(c->stream);
  c->allocs.clear();
  c->alloc_bytes.clear();
  for (int q = 0; q < 3; q++) {
    if (c->fork_ev[q]) cudaEventDestroy(c->fork_ev[q]);
    if (c->join_ev[q]) cudaEventDestroy(c->join_ev[q]);
  }
  if (c->side) cudaStreamDestroy(c->side);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return MD_OK;
}

int md_ctx_stream(md_ctx* c, void** stream) {
  if (!c || !stream) return set_err(c, MD_ERR_INVALID, "null argument");
  *stream = (void*)c->stream;
  return MD_OK;
}

int md_ctx_device_bytes(const md_ctx* c, int64_t* bytes) {
  if (!c || !bytes) return MD_ERR_INVALID;
  *bytes = c->bytes;
  return MD_OK;
}

int md_set_particles(md_ctx* c, const double* rMag, const double* rHydr) {
  if (!c || !rMag) return set_err(c, MD_ERR_INVALID, "null argument");
  std::string e;
  mdh::Props p;
  int st = mdh::make_props(c->cfg, rMag, rHydr, c->n, &p, &e);
  if (st) return set_err(c, st, "%s", e.c_str());
  if ((st = count_pairs(c))) return st;
  c->props = p;
  c->L = p.lBox;
  const size_t N = (size_t)c->n;
  std::vector<double> mu(N), rm(N), izt(N), ivol(N);
  for (size_t i = 0; i < N; i++) {
    mu[i] = p.magMom[i] / p.muMax;
    rm[i] = p.rMag[i] / c->L;
    izt[i] = 1.0 / p.zetaTrans[i];
    ivol[i] = 1.0 / p.volMag[i];
  }
  CK(c, cudaMemcpyAsync(c->magMom_u, mu.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->rMag_u, rm.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->invZt, izt.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->velEa1, p.velEa1.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->velEa2, p.velEa2.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->zetaR, p.zetaRot.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->zetaT, p.zetaTrans.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaMemcpyAsync(c->invVol, ivol.data(), 8 * N, cudaMemcpyHostToDevice, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  c->have_particles = true;
  c->have_ewald = false;
  c->list_valid = false;
  c->cur_dt = -1;
  invalidate_graph(c);
  return MD_OK;
}

int md_get_box(const md_ctx* c, double* lBox) {
  if (!c || !lBox) return MD_ERR_INVALID;
  *lBox = c->L;
  return MD_OK;
}

int md_set_box(md_ctx* c, double lBox) {
  if (!c || !(lBox > 0) || !c->have_particles) return set_err(c, MD_ERR_INVALID, "bad box or particles not set");
  if (int st = count_pairs(c)) return st;
  c->L = lBox;
  c->props.lBox = lBox;
  std::vector<double> rm(c->n);
  for (int64_t i = 0; i < c->n; i++) rm[i] = c->props.rMag[i] / lBox;
  CK(c, cudaMemcpy(c->rMag_u, rm.data(), 8 * c->n, cudaMemcpyHostToDevice));
  c->cur_dt = -1;  // the integrator's constants hold rMag / L
  c->have_ewald = false;
  c->list_valid = false;
  invalidate_graph(c);
  return MD_OK;
}

// Device-side address of a host buffer of `bytes` bytes that kernels may
// read and write directly (page-locked memory mapped into the device's
// address space, its first and last element in one contiguous mapping),
// else null (pageable or partly registered memory: copied by the copy
// engines).
static double* mapped_addr(const double* h, size_t bytes) {
  auto dev = [](const void* q) -> char* {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, q) != cudaSuccess) {
      cudaGetLastError();  // not a CUDA allocation: no sticky error
      return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? (char*)a.devicePointer : nullptr;
  };
  if (bytes < sizeof(double)) return nullptr;
  const char* last = (const char*)h + bytes - sizeof(double);
  char* d0 = dev(h);
  char* d1 = d0 ? dev(last) : nullptr;
  return (d1 && d1 - d0 == last - (const char*)h) ? (double*)d0 : nullptr;
}

// The copies and checks of md_state_upload, queued on the stream.  Mapped
// host buffers come in through one kernel that also does the displacement
// check; others through three copies and the check's own launch.
static int enqueue_upload(md_ctx* c, const double* pos, const double* mm, const double* ea, int reset) {
  const size_t B = 24 * (size_t)c->n;
  const double *dp = mapped_addr(pos, B), *dm = mapped_addr(mm, B), *de = mapped_addr(ea, B);
  const bool direct = dp && dm && de;
  if (direct) {
    launch_state_in(c->stream, (int)c->n, dp, dm, de, c->pos, c->mm, c->ea, c->list_valid ? c->xbuild : nullptr, c->L,
                    &c->sc->flags);
  } else {
    CK(c, cudaMemcpyAsync(c->pos, pos, B, cudaMemcpyHostToDevice, c->stream));
    CK(c, cudaMemcpyAsync(c->mm, mm, B, cudaMemcpyHostToDevice, c->stream));
    CK(c, cudaMemcpyAsync(c->ea, ea, B, cudaMemcpyHostToDevice, c->stream));
  }
  if (reset || !c->have_state) {
    CK(c, cudaMemcpyAsync(c->truePos, c->pos, B, cudaMemcpyDeviceToDevice, c->stream));
    CK(c, cudaMemcpyAsync(c->posRef, c->pos, B, cudaMemcpyDeviceToDevice, c->stream));
  }
  if (c->list_valid) {
    // same particles: rebuild on the next step only if they moved beyond the skin
    if (!direct) launch_disp_check(c->stream, (int)c->n, c->pos, c->xbuild, c->L, &c->sc->flags);
  } else if (int st = force_rebuild(c)) {
    return st;
  }
  c->have_state = true;
  c->have_geometry = false;
  return MD_OK;
}

int md_state_upload(md_ctx* c, const double* pos, const double* mm, const double* ea, int reset) {
  if (!c || !pos || !mm || !ea) return set_err(c, MD_ERR_INVALID, "null argument");
  if (int st = enqueue_upload(c, pos, mm, ea, reset)) return st;
  CK(c, cudaStreamSynchronize(c->stream));
  return MD_OK;
}

int md_state_download(md_ctx* c, double* pos, double* mm, double* ea) {
  if (!c) return set_err(c, MD_ERR_INVALID, "null context");
  const size_t B = 24 * (size_t)c->n;
  if (pos) CK(c, cudaMemcpyAsync(pos, c->pos, B, cudaMemcpyDeviceToHost, c->stream));
  if (mm) CK(c, cudaMemcpyAsync(mm, c->mm, B, cudaMemcpyDeviceToHost, c->stream));
  if (ea) CK(c, cudaMemcpyAsync(ea, c->ea, B, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return MD_OK;
}

int md_set_time(md_ctx* c, double t, int64_t step) {
  if (!c) return set_err(c, MD_ERR_INVALID, "null context");
  CK(c, cudaStreamSynchronize(c->stream));
  DevScalars h;
  CK(c, cudaMemcpy(&h, c->sc, sizeof h, cudaMemcpyDeviceToHost));
  h.time = t;
  h.step = step;
  CK(c, cudaMemcpy(c->sc, &h, sizeof h, cudaMemcpyHostToDevice));
  return MD_OK;
}

int md_get_time(const md_ctx* cc, double* t, int64_t* step) {
  md_ctx* c = const_cast<md_ctx*>(cc);
  if (!c) return MD_ERR_INVALID;
  DevScalars h;
  CK(c, cudaStreamSynchronize(c->stream));
  CK(c, cudaMemcpy(&h, c->sc, sizeof h, cudaMemcpyDeviceToHost));
  if (t) *t = h.time;
  if (step) *step = h.step;
  return MD_OK;
}

int md_ewald_params(md_ctx* c, double rc, double* alpha, double* rc_out, int64_t* kc, double* errF, double* errT) {
  if (!c || !c->have_particles) return set_err(c, MD_ERR_INVALID, "particles not set");
  mdh::EwaldModel m = mdh::ewald_model(c->cfg, c->props);
  double a = 0, kraw = 0;
  int64_t k = 0;
  if (rc <= 0) {
    rc = mdh::choose_rc(c->cfg, m, c->n, &a, &k, tc_kc_bound(c));
    kraw = (double)k;
  } else {
    if (rc > 0.5 * c->L * (1 + 1e-12)) return set_err(c, MD_ERR_INVALID, "rc must not exceed L/2");
    if (!mdh::ewald_for_rc(c->cfg, m, rc, &a, &kraw))
      return set_err(c, MD_ERR_INVALID, "alpha for the error tolerance not found");
    k = (int64_t)std::floor(kraw + 0.5);
  }
  if (alpha) *alpha = a;
  if (rc_out) *rc_out = rc;
  if (kc) *kc = k;
  mdh::predicted_errors(c->cfg, m, a, rc, (double)k, errF, errT);
  return MD_OK;
}

int md_ewald_params_host(const md_config* cfg, int64_t n, const double* rMag, const double* rHydr, double rc,
                         double* alpha, double* rc_out, int64_t* kc, double* errF, double* errT, double* lBox) {
  if (!cfg || !rMag || n < 2) return set_err(nullptr, MD_ERR_INVALID, "bad arguments");
  std::string e;
  mdh::Props p;
  int st = mdh::make_props(*cfg, rMag, rHydr, n, &p, &e);
  if (st) return set_err(nullptr, st, "%s", e.c_str());
  mdh::EwaldModel m = mdh::ewald_model(*cfg, p);
  double a = 0, kraw = 0;
  int64_t k = 0;
  if (rc <= 0) {
    rc = mdh::choose_rc(*cfg, m, n, &a, &k, cfg->precision == MD_PREC_MIXED ? md::kspace_tc_max_kc() : 0);
  } else {
    if (rc > 0.5 * p.lBox * (1 + 1e-12)) return set_err(nullptr, MD_ERR_INVALID, "rc must not exceed L/2");
    if (!mdh::ewald_for_rc(*cfg, m, rc, &a, &kraw))
      return set_err(nullptr, MD_ERR_INVALID, "alpha for the error tolerance not found");
    k = (int64_t)std::floor(kraw + 0.5);
  }
  if (alpha) *alpha = a;
  if (rc_out) *rc_out = rc;
  if (kc) *kc = k;
  if (lBox) *lBox = p.lBox;
  mdh::predicted_errors(*cfg, m, a, rc, (double)k, errF, errT);
  return MD_OK;
}

int md_set_ewald(md_ctx* c, double alpha, double rc, int64_t kc) {
  if (!c || !c->have_particles) return set_err(c, MD_ERR_INVALID, "particles not set");
  if (!(alpha > 0) || !(rc > 0) || rc > 0.5 * c->L * (1 + 1e-12) || kc < 1 || kc > 96)
    return set_err(c, MD_ERR_INVALID, "bad Ewald parameters (alpha>0, 0<rc<=L/2, 1<=kc<=96)");
  if (!fp64(c) && kscatter_smem((int)kc) == 0) return set_err(c, MD_ERR_UNSUPPORTED, "kc too large for shared memory");
  invalidate_graph(c);
  CK(c, cudaStreamSynchronize(c->stream));
  if (int st = count_pairs(c)) return st;
  c->alpha = alpha;
  c->rc = rc;
  c->kc = kc;
  c->list_valid = false;
  const double ab = alpha * c->L;
  const double w = std::pow(c->cfg.my_pi / ab, 2.0);
  c->klist = mdh::build_klist((int)kc, w);
  c->grid = cell_grid(rc / c->L, c->n, fp64(c));
  if (!fp64(c)) segment_chunks(c->klist, c->n, (int)kc, num_sms(c->device), &c->chunk, &c->nchunk);
  // (re)allocate Ewald-sized buffers
  const int ncell = c->grid.ncell;
  if (ncell + 1 > c->ncell_cap) {
    dfree(c, c->count);
    dfree(c, c->cell_start);
    c->count = nullptr;
    c->cell_start = nullptr;
    int st;
    if ((st = dalloc(c, &c->count, 4 * (size_t)(ncell + 1)))) return st;
    if ((st = dalloc(c, &c->cell_start, 4 * (size_t)(ncell + 1)))) return st;
    // the cell fill counters are zero between builds (the build leaves them so)
    CK(c, cudaMemset(c->count, 0, 4 * (size_t)(ncell + 1)));
    c->ncell_cap = ncell + 1;
  }
  if (c->grid.ncx == 1) {
    int h[2] = {0, (int)c->n};
    CK(c, cudaMemcpy(c->cell_start, h, sizeof h, cudaMemcpyHostToDevice));
  }
  const size_t nk = (size_t)c->klist.nk, nseg = c->klist.seg.size();
  const size_t nks = (size_t)c->klist.nk_scat, nrseg = c->klist.rseg.size();
  const size_t need = std::max(std::max(nk, nseg), std::max(nks, nrseg)) + 2;
  if (need > c->ksize_cap) {
    void* old[] = {c->kseg, c->koff, c->ek, c->eS, c->Sfull, c->rseg, c->rowpos, c->chunks};
    for (void* p : old) dfree(c, p);
    const size_t cap = need;
    int st;
    if ((st = dalloc(c, &c->ek, sizeof(double) * cap))) return st;
    if ((st = dalloc(c, &c->Sfull, sizeof(double2) * cap))) return st;
    if (!fp64(c)) {  // row segments of the CUDA-core kernels
      if ((st = dalloc(c, &c->kseg, sizeof(KSeg) * cap))) return st;
      if ((st = dalloc(c, &c->koff, sizeof(int) * cap))) return st;
      if ((st = dalloc(c, &c->eS, 8 * cap))) return st;
      if ((st = dalloc(c, &c->rseg, sizeof(KSeg) * cap))) return st;
      if ((st = dalloc(c, &c->rowpos, sizeof(int) * cap))) return st;
      if ((st = dalloc(c, &c->chunks, sizeof(int2) * cap))) return st;
    }
    c->ksize_cap = cap;
  }
  const size_t sp = nk * (size_t)c->nchunk;
  if (!fp64(c) && sp > c->spart_cap) {
    dfree(c, c->Spart);
    c->Spart = nullptr;
    int st;
    if ((st = dalloc(c, &c->Spart, sizeof(double2) * sp))) return st;
    c->spart_cap = sp;
  }
  const size_t pt = (size_t)3 * (c->kc + 1) * c->n * 2 * tsz(c);
  if (pt > c->ptab_cap) {
    dfree(c, c->ptab);
    c->ptab = nullptr;
    int st;
    if ((st = dalloc(c, &c->ptab, pt))) return st;
    c->ptab_cap = pt;
  }
  if (!fp64(c) && c->nchunk > c->musum_cap) {
    dfree(c, c->musum_part);
    c->musum_part = nullptr;
    int st;
    if ((st = dalloc(c, &c->musum_part, 24 * (size_t)c->nchunk))) return st;
    c->musum_cap = c->nchunk;
  }
  CK(c, cudaMemcpy(c->ek, c->klist.ek.data(), sizeof(double) * nk, cudaMemcpyHostToDevice));
  if (!fp64(c)) {
    CK(c, cudaMemcpy(c->kseg, c->klist.seg.data(), sizeof(KSeg) * nseg, cudaMemcpyHostToDevice));
    CK(c, cudaMemcpy(c->koff, c->klist.koff.data(), sizeof(int) * nseg, cudaMemcpyHostToDevice));
    CK(c, cudaMemcpy(c->rseg, c->klist.rseg.data(), sizeof(KSeg) * nrseg, cudaMemcpyHostToDevice));
    CK(c, cudaMemcpy(c->rowpos, c->klist.rowpos.data(), sizeof(int) * nk, cudaMemcpyHostToDevice));
    // the padding entries of the scatter layout are never written: zero
    CK(c, cudaMemset(c->eS, 0, 8 * nks));
    CK(c, cudaMemcpy(c->chunks, c->klist.chunks.data(), sizeof(int) * c->klist.chunks.size(), cudaMemcpyHostToDevice));
  }
  if (int st = setup_engine(c)) return st;
  {
    // k-space self-interaction: B_i holds -cflux sum_k e(k) (n . mu_i) n of
    // each particle's own moment (the k list's e(k) covers the half space)
    double K[6] = {0, 0, 0, 0, 0, 0};
    for (size_t k = 0; k < c->klist.ek.size(); k++) {
      if (!c->klist.kreal[k]) continue;
      const double e = c->klist.ek[k], nx = c->klist.kx[k], ny = c->klist.ky[k], nz = c->klist.kz[k];
      K[0] += e * nx * nx;
      K[1] += e * ny * ny;
      K[2] += e * nz * nz;
      K[3] += e * nx * ny;
      K[4] += e * nx * nz;
      K[5] += e * ny * nz;
    }
    for (int q = 0; q < 6; q++) c->kself[q] = 4.0 * c->cfg.my_pi * K[q];
  }
  {
    int st = alloc_nbr(c, mdh::list_entries(c->n, rc / c->L * (1.0 + c->skin_frac)));
    if (st) return st;
  }
  update_strong(c);
  if (c->strong_w4sq > 0.f && !c->cfg.ENABLE_COATING_POT)
    if (int st = alloc_strong(c, strong_entries(c))) return st;
  if (int st = force_rebuild(c)) return st;
  c->have_ewald = true;
  c->have_geometry = false;
  return MD_OK;
}

// The allocations of md_ctx_create and md_set_ewald, and of the records.
double mdi_packed_ctx_bytes(const md_config* cfg, int64_t n, const double* rMag, double alpha, double rc,
                                       int64_t kc, int64_t steps) {
  mdh::Props p;
  std::string e;
  if (mdh::make_props(*cfg, rMag, nullptr, n, &p, &e)) return -1.0;
  int dev = 0;
  cudaGetDevice(&dev);
  const int nsm = num_sms(dev);
  const double N = (double)n, L = p.lBox, rl = rc * (1.0 + kSkinFrac);
  const mdh::KList k = mdh::build_klist((int)kc, std::pow(cfg->my_pi / (alpha * L), 2.0));
  const size_t ks = std::max(std::max((size_t)k.nk, k.seg.size()), std::max((size_t)k.nk_scat, k.rseg.size())) + 2;
  int chunk = 0, nchunk = 0;
  segment_chunks(k, n, (int)kc, nsm, &chunk, &nchunk);
  double b = 677.0 * N + 4096;                                        // state, stages and work arrays
  b += 8.0 * (cell_grid(rc / L, n, false).ncell + 1);                 // cells
  b += 4.0 * (double)mdh::list_entries(n, rl / L);                    // neighbour list
  if (!cfg->ENABLE_COATING_POT)                                       // strong list and its sums
    b += (sizeof(int2) + 96.0) * (4096 + 2.0 * strong_estimate(p, L, rl, kStrongTheta));
  b += (48.0 + 2 * sizeof(KSeg)) * (double)ks + 16.0 * (double)k.nk * nchunk + 24.0 * (kc + 1) * N;  // k vectors, phases
  if (md::kspace_tc_supported((int)kc)) {
    std::set<std::pair<int, int>> rows;
    for (int q = 0; q < k.nk; q++)
      if (k.kreal[q]) rows.insert({k.kz[q], k.ky[q]});
    const int R = (int)rows.size();
    const md::TcShape t = md::kspace_tc_shape((int)kc, (int)n, R, nsm, -1, 1);
    b += 8.0 * R + 16.0 * md::kspace_tc_rows_pad(R) + 4.0 * R * (2 * kc + 1);
    b += 4.0 * ((double)t.nchunk * t.mt * t.ns * 128 + (double)md::kspace_tc_image_floats((int)kc, t.nt_full) +
                (double)md::kspace_tc_image_floats((int)kc, t.nt_field) +
                (double)md::kspace_tc_bimg_floats((int)kc, t.nsb)) +
         8.0 * (double)md::kspace_tc_tblk_entries((int)kc, t.nsb);
    nchunk = std::max(nchunk, t.nchunk);
  }
  b += 24.0 * nchunk;
  return b + 64.0 * (steps + 1024);
}

int md_set_kspace_engine(md_ctx* c, int engine) {
  if (!c || engine < MD_KSPACE_AUTO || engine > MD_KSPACE_TC) return set_err(c, MD_ERR_INVALID, "bad k-space engine");
  if (engine == MD_KSPACE_TC && fp64(c))
    return set_err(c, MD_ERR_UNSUPPORTED, "the tensor-core k space is part of the mixed path");
  if (engine == MD_KSPACE_TC && c->have_ewald && !md::kspace_tc_supported((int)c->kc))
    return set_err(c, MD_ERR_UNSUPPORTED, "kc too large for the tensor-core k space");
  invalidate_graph(c);
  CK(c, cudaStreamSynchronize(c->stream));
  c->kengine = engine;
  // the per-step operand images of a newly chosen engine come with the next full evaluation
  c->have_geometry = false;
  return c->have_ewald ? setup_engine(c) : MD_OK;
}

int md_kspace_engine_active(const md_ctx* c, int* tensor_cores) {
  if (!c || !tensor_cores) return MD_ERR_INVALID;
  *tensor_cores = c->tc_rows > 0 ? 1 : 0;
  return MD_OK;
}

int md_kspace_engine_used(const md_ctx* c, int* engine) {
  if (!c || !engine) return MD_ERR_INVALID;
  // in the order of launch_kspace
  *engine = !c->have_ewald ? 0
            : c->rw_T > 0  ? MD_KSPACE_ROWS
            : c->gm_M > 0  ? MD_KSPACE_MESH
            : c->tc_rows > 0 ? MD_KSPACE_TC
                             : MD_KSPACE_SIMT;
  return MD_OK;
}

int md_set_kspace_tiling(md_ctx* c, int ring, int waves) {
  if (!c || ring < -1 || ring > 5 || waves < 1 || waves > 4) return set_err(c, MD_ERR_INVALID, "bad k-space tiling");
  invalidate_graph(c);
  CK(c, cudaStreamSynchronize(c->stream));
  c->tc_ring = ring;
  c->tc_waves = waves;
  c->have_geometry = false;  // the per-step operands come with the next full evaluation
  return c->have_ewald ? setup_engine(c) : MD_OK;
}

int md_get_kspace_tiling(const md_ctx* c, int* ring, int* waves, int* chunk) {
  if (!c) return MD_ERR_INVALID;
  if (ring) *ring = c->tc_ring;
  if (waves) *waves = c->tc_waves;
  if (chunk) *chunk = c->tc_rows > 0 ? c->tcs.chunk : 0;
  return MD_OK;
}

int md_compute_interactions(md_ctx* c, double* B, double* F, double* P3) {
  NvtxRange nv("md_compute_interactions");
  int st = check_ready(c, true);
  if (st) return st;
  if ((st = force_rebuild(c))) return st;
  const size_t Bz = 24 * (size_t)c->n;
  const int nb = int_blocks((int)c->n);
  std::vector<double> pp(3 * (size_t)nb);
  DevScalars h;
  c->launches = 0;
  // evaluated again when the strong list did not fit its estimate: grown and
  // built anew, so the returned result has its strong pairs in FP64
  for (int pass = 0; pass < 2; pass++) {
    c->launches += issue_interactions(c);
    IntParams ip = int_params(c, 0.0, c->Br, c->Bk);
    if (!fp64(c)) ip.mexact = c->mm;
    c->launches += launch_combine(c->stream, ip, c->Bout, c->Fout, c->obs_part, 1 + pass, fp64(c));
    CK(c, cudaGetLastError());
    CK(c, cudaMemcpyAsync(&h, c->sc, sizeof h, cudaMemcpyDeviceToHost, c->stream));
    CK(c, cudaMemcpyAsync(pp.data(), c->obs_part, 8 * pp.size(), cudaMemcpyDeviceToHost, c->stream));
    if (B) CK(c, cudaMemcpyAsync(B, c->Bout, Bz, cudaMemcpyDeviceToHost, c->stream));
    if (F) CK(c, cudaMemcpyAsync(F, c->Fout, Bz, cudaMemcpyDeviceToHost, c->stream));
    CK(c, cudaStreamSynchronize(c->stream));
    const bool again = pass == 0 && strong_active(c) && h.flags.soverflow && !h.flags.overflow;
    if ((st = handle_overflow(c, h.flags))) return st;
    if (!again) break;
  }
  if (P3) {
    double s[3] = {0.0, 0.0, 0.0};
    for (size_t b = 0; b < pp.size() / 3; b++)
      for (int q = 0; q < 3; q++) s[q] += pp[3 * b + q];
    const double sc = c->L * F_unit(c) / 2.0;
    for (int q = 0; q < 3; q++) P3[q] = s[q] * sc;
  }
  return MD_OK;
}

int md_compute_field(md_ctx* c, const double* mm, double* B) {
  NvtxRange nv("md_compute_field");
  int st = check_ready(c, true);
  if (st) return st;
  if (!mm) return set_err(c, MD_ERR_INVALID, "null moment directions");
  if (!c->have_geometry) return set_err(c, MD_ERR_INVALID, "call md_compute_interactions first");
  CK(c, cudaMemcpyAsync(c->tmpmm, mm, 24 * (size_t)c->n, cudaMemcpyHostToDevice, c->stream));
  SortedView s = sorted_view(c);
  c->launches = launch_set_mu(c->stream, (int)c->n, c->tmpmm, c->magMom_u, c->rMag_u, s, fp64(c));
  c->launches += issue_field(c);
  IntParams ip = int_params(c, 0.0, c->Br2, c->Bk2);
  if (!fp64(c)) ip.mexact = c->tmpmm;
  c->launches += launch_combine(c->stream, ip, c->Bout, nullptr, nullptr, 0, fp64(c));
  CK(c, cudaGetLastError());
  if (B) CK(c, cudaMemcpyAsync(B, c->Bout, 24 * (size_t)c->n, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return MD_OK;
}

int md_set_noise(md_ctx* c, int mode, uint64_t seed) {
  if (!c || mode < 0 || mode > 2) return set_err(c, MD_ERR_INVALID, "bad noise mode");
  c->noise = mode;
  c->seed = seed;
  invalidate_graph(c);
  return MD_OK;
}

}  // extern "C"

// Room for `extra` more step records.  The host keeps an upper bound of the
// device's record count (records issued since it was last read or cleared)
// and reads the device only when the bound would pass the capacity, so a
// step does not wait on a device read.
int ensure_records(md_ctx* c, int64_t extra) {
  if (c->nrec_bound + extra <= c->rec_cap) {
    c->nrec_bound += extra;
    return MD_OK;
  }
  long long nrec = 0;
  CK(c, cudaStreamSynchronize(c->stream));
  CK(c, cudaMemcpy(&nrec, &c->sc->nrec, sizeof nrec, cudaMemcpyDeviceToHost));
  c->nrec_bound = nrec + extra;
  if (nrec + extra <= c->rec_cap) return MD_OK;
  long long cap = std::max<long long>(1024, 2 * (nrec + extra));
  double* nr = nullptr;
  int st = dalloc(c, &nr, 64 * (size_t)cap);
  if (st) return st;
  if (c->records && nrec > 0) CK(c, cudaMemcpy(nr, c->records, 64 * (size_t)nrec, cudaMemcpyDeviceToDevice));
  dfree(c, c->records);
  c->records = nr;
  c->rec_cap = cap;
  invalidate_graph(c);
  return MD_OK;
}

// DefThermFluct prefactors (src/simulation.cpp:563-603) and the other
// per-particle constants of the integrator, computed on the device for this
// dt (queued on the stream; the adaptive solvers change dt every step).
int prepare_dt(md_ctx* c, double dt) {
  if (dt == c->cur_dt) return MD_OK;
  const md_config& g = c->cfg;
  const double kt = 2.0 * g.kB * g.temp / dt;
  const double kb = 2.0 * g.kB * g.temp * g.magDamp / (g.gyroMr * g.satMag * dt);
  cudaGetLastError();  // an earlier call's error was reported there
  launch_int_consts(c->stream, (int)c->n, g.ENABLE_THERM_TORQUE ? kt : 0.0, g.ENABLE_THERM_FIELD ? kb : 0.0,
                    g.ENABLE_THERM_FORCE ? kt : 0.0, c->zetaR, c->zetaT, c->invVol, c->invZt, c->velEa1, c->velEa2,
                    c->magMom_u, c->rMag_u, c->sTB, c->cA, c->cB, fp64(c));
  CK(c, cudaGetLastError());
  c->cur_dt = dt;
  invalidate_graph(c);
  return MD_OK;
}

// Captures k steps as one graph; *launches: its kernels.
static int capture_steps(md_ctx* c, int k, double dt, cudaGraph_t* graph, cudaGraphExec_t* exec, int64_t* launches) {
  *launches = 0;
  CK(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
  for (int s = 0; s < k; s++) *launches += issue_step(c, dt, s > 0, s < k - 1);
  cudaError_t e = cudaStreamEndCapture(c->stream, graph);
  if (e != cudaSuccess) return set_err(c, MD_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
  CK(c, cudaGraphInstantiate(exec, *graph, 0));
  return MD_OK;
}

// Between two graphs lie ~3.4 us, between a graph's own steps ~0.7: a run that has
// shown to be long (its capture, ~1 ms, then pays) goes on in graphs of several
// steps.  N = 512 51.2 -> 47.4, N = 1000 59.5 -> 55.6, N = 3001 91.6 -> 87.7, N = 8192
// 153.6 -> 148.9, N = 32768 585.6 -> 579.9 us per step.
constexpr int kGraphSteps = 8, kGraphAfter = 128;

// md_step's work queued on the stream (no synchronisation).
static int enqueue_steps(md_ctx* c, int64_t nsteps, double dt, const double* xi) {
  int st = check_ready(c, true);
  if (st) return st;
  if (nsteps < 0 || !(dt > 0)) return set_err(c, MD_ERR_INVALID, "bad nsteps or dt");
  if (c->noise == MD_NOISE_UPLOADED && !xi) return set_err(c, MD_ERR_INVALID, "uploaded noise needs xi");
  if (nsteps == 0) return MD_OK;
  if ((st = prepare_dt(c, dt))) return st;
  if ((st = ensure_records(c, nsteps))) return st;
  if (c->noise == MD_NOISE_UPLOADED) {
    c->launches = 0;
    for (int64_t s = 0; s < nsteps; s++) {
      CK(c, cudaMemcpyAsync(c->xi, xi + (size_t)s * 9 * c->n, 72 * (size_t)c->n, cudaMemcpyHostToDevice, c->stream));
      c->launches += issue_step(c, dt);
    }
    CK(c, cudaGetLastError());
  } else {
    if (!c->graph_valid) {
      if ((st = capture_steps(c, 1, dt, &c->graph, &c->gexec, &c->launches_1))) return st;
      c->graph_valid = true;
    }
    c->launches = 0;
    int64_t s = 0;
    while (s < nsteps) {
      if (nsteps - s >= kGraphSteps && (c->gexec_n || c->replays >= kGraphAfter) && !c->prof) {
        if (!c->gexec_n && (st = capture_steps(c, kGraphSteps, dt, &c->graph_n, &c->gexec_n, &c->launches_n))) return st;
        CK(c, cudaGraphLaunch(c->gexec_n, c->stream));
        c->launches += c->launches_n;
        s += kGraphSteps;
      } else {
        CK(c, cudaGraphLaunch(c->gexec, c->stream));
        c->launches += c->launches_1;
        c->replays++;
        s++;
      }
    }
  }
  c->have_geometry = true;
  return MD_OK;
}

extern "C" {

int md_step(md_ctx* c, int64_t nsteps, double dt, const double* xi) {
  NvtxRange nv("md_step");
  if (int st = enqueue_steps(c, nsteps, dt, xi)) return st;
  return read_err_word(c);
}

int md_step_io(md_ctx* c, const double* pos, const double* mm, const double* ea, int64_t nsteps, double dt,
               double* pos_out, double* mm_out, double* ea_out) {
  NvtxRange nv("md_step_io");
  if (!c || !pos || !mm || !ea || !pos_out || !mm_out || !ea_out) return set_err(c, MD_ERR_INVALID, "null argument");
  if (c->noise == MD_NOISE_UPLOADED) return set_err(c, MD_ERR_INVALID, "md_step_io draws its noise (Philox or off)");
  int st = enqueue_upload(c, pos, mm, ea, 0);
  if (!st) st = enqueue_steps(c, nsteps, dt, nullptr);
  if (st) {
    cudaStreamSynchronize(c->stream);
    return st;
  }
  const size_t B = 24 * (size_t)c->n;
  double *op = mapped_addr(pos_out, B), *om = mapped_addr(mm_out, B), *oe = mapped_addr(ea_out, B);
  if (op && om && oe) {
    // mapped host buffers: written by one kernel
    launch_state_out(c->stream, (int)c->n, c->pos, c->mm, c->ea, op, om, oe);
  } else {
    CK(c, cudaMemcpyAsync(pos_out, c->pos, B, cudaMemcpyDeviceToHost, c->stream));
    CK(c, cudaMemcpyAsync(mm_out, c->mm, B, cudaMemcpyDeviceToHost, c->stream));
    CK(c, cudaMemcpyAsync(ea_out, c->ea, B, cudaMemcpyDeviceToHost, c->stream));
  }
  return read_err_word(c);
}

// Butcher rows of the reference's solvers (src/simulation.cpp:721-867):
// weights of k_0..k_s for stage s + 1, error weights, solution weights.
namespace {
struct Tableau {
  int stages;
  double power;
  double a[7][7];
  double e[7];
  double b[7];
  int nb;         // solution weights b[0..nb)
  bool last_is_solution;  // Bogacki-Shampine: the solution is the last stage's coordinates
};

const Tableau& tableau(int solver) {
  static const Tableau he = {2, 1.0 / 2.0, {{1.0}}, {0.5, -0.5}, {0.5, 0.5}, 2, false};
  static const Tableau bs = {4,
                             1.0 / 3.0,
                             {{1.0 / 2.0}, {0, 3.0 / 4.0}, {2.0 / 9.0, 1.0 / 3.0, 4.0 / 9.0}},
                             {-5.0 / 72.0, 1.0 / 12.0, 1.0 / 9.0, -1.0 / 8.0},
                             {},
                             0,
                             true};
  static const Tableau dp = {7,
                             1.0 / 5.0,
                             {{1.0 / 5.0},
                              {3.0 / 40.0, 9.0 / 40.0},
                              {44.0 / 45.0, -56.0 / 15.0, 32.0 / 9.0},
                              {19372.0 / 6561.0, -25360.0 / 2187.0, 64448.0 / 6561.0, -212.0 / 729.0},
                              {9017.0 / 3168.0, -355.0 / 33.0, 46732.0 / 5247.0, 49.0 / 176.0, -5103.0 / 18656.0},
                              {35.0 / 384.0, 0, 500.0 / 1113.0, 125.0 / 192.0, -2187.0 / 6784.0, 11.0 / 84.0}},
                             {71.0 / 57600.0, 0, -71.0 / 16695.0, 71.0 / 1920.0, -17253.0 / 339200.0, 22.0 / 525.0,
                              -1.0 / 40.0},
                             {35.0 / 384.0, 0, 500.0 / 1113.0, 125.0 / 192.0, -2187.0 / 6784.0, 11.0 / 84.0},
                             6,
                             false};
  return solver == 1 ? bs : (solver == 2 ? dp : he);
}
}  // namespace

int md_step_adaptive(md_ctx* c, int64_t max_steps, double t_end, double* dt_io, const double* xi,
                     int64_t* steps_done) {
  NvtxRange nv("md_step_adaptive");
  int st = check_ready(c, true);
  if (st) return st;
  if (steps_done) *steps_done = 0;
  if (max_steps < 0 || !dt_io || !(*dt_io > 0)) return set_err(c, MD_ERR_INVALID, "bad max_steps or dt");
  if (c->noise == MD_NOISE_UPLOADED && !xi && max_steps > 0)
    return set_err(c, MD_ERR_INVALID, "uploaded noise needs xi");
  const int solver = (int)c->cfg.SOLVER;
  if (solver < 0 || solver > 2) return set_err(c, MD_ERR_INVALID, "SOLVER must be 0, 1 or 2");
  const Tableau& tb = tableau(solver);
  const double absTol = c->cfg.absTol, dtMin = c->cfg.deltaTmin, dtMax = c->cfg.deltaTmax;
  const size_t n3t = 3 * (size_t)c->n * tsz(c);
  for (int q = 0; q < tb.stages; q++) {
    if (!c->rk_km[q] && (st = dalloc(c, &c->rk_km[q], n3t))) return st;
    if (!c->rk_ke[q] && (st = dalloc(c, &c->rk_ke[q], n3t))) return st;
  }
  if (!c->rk_cm && (st = dalloc(c, &c->rk_cm, n3t))) return st;
  if (!c->rk_ce && (st = dalloc(c, &c->rk_ce, n3t))) return st;
  if ((st = ensure_records(c, max_steps))) return st;
  double t = 0;
  int64_t stepno = 0;
  if ((st = md_get_time(c, &t, &stepno))) return st;
  RKStage q{};
  for (int j = 0; j < 7; j++) {
    q.km[j] = c->rk_km[j];
    q.ke[j] = c->rk_ke[j];
  }
  q.cm = c->rk_cm;
  q.ce = c->rk_ce;
  q.errmax = &c->sc->errmax;
  q.sTB = c->sTB;
  int64_t done = 0;
  c->launches = 0;
  while (done < max_steps && t <= t_end) {
    const double dt0 = *dt_io;
    if ((st = prepare_dt(c, dt0))) return st;
    if (c->noise == MD_NOISE_UPLOADED)
      CK(c, cudaMemcpyAsync(c->xi, xi + (size_t)done * 9 * c->n, 72 * (size_t)c->n, cudaMemcpyHostToDevice,
                            c->stream));
    c->launches += issue_interactions(c, dt0, true);
    bool cond = true, noFailed = true, first = true;
    double nf = 1.0, used = dt0;
    while (cond) {
      const double dt = *dt_io;
      q.nf = nf;
      for (int s = 0; s < tb.stages; s++) {
        const bool start_field = s == 0 && first;  // later: the field last evaluated
        q.p = int_params(c, dt, start_field ? c->Br : c->Br2, start_field ? c->Bk : c->Bk2);
        q.s = s;
        q.last = s == tb.stages - 1;
        for (int j = 0; j < 7; j++) {
          q.a[j] = q.last ? 0.0 : tb.a[s][j];
          q.e[j] = tb.e[j];
        }
        if (q.last) CK(c, cudaMemsetAsync(&c->sc->errmax, 0, sizeof(unsigned long long), c->stream));
        c->launches += launch_rk_stage(c->stream, q, fp64(c));
        if (!q.last) c->launches += issue_field(c);
      }
      unsigned long long bits = 0;
      CK(c, cudaMemcpyAsync(&bits, &c->sc->errmax, sizeof bits, cudaMemcpyDeviceToHost, c->stream));
      CK(c, cudaStreamSynchronize(c->stream));
      double emax;
      std::memcpy(&emax, &bits, sizeof emax);
      const double error = dt * emax;
      used = dt;
      // AdjustTimeStep (src/simulation.cpp:912-951), including its clamp:
      // min(., deltaTmax) is overwritten by max(., deltaTmin)
      double tnew;
      if (error > absTol) {
        if (noFailed) {
          noFailed = false;
          tnew = std::max(dtMin, dt * std::max(0.1, 0.9 * std::pow(absTol / error, tb.power)));
        } else {
          tnew = std::max(dtMin, dt * 0.5);
        }
        nf *= std::sqrt(tnew / dt);
        if (tnew == dt) {
          // the reference would retry the same step forever (deltaTmin reached)
          return set_err(c, MD_ERR_INVALID, "step rejected at deltaTmin = %g s (error %g > absTol %g)", dt, error,
                         absTol);
        }
      } else {
        tnew = noFailed ? dt * std::min(std::max(0.9 * std::pow(absTol / error, tb.power), 0.2), 5.0) : dt;
        cond = false;
      }
      *dt_io = std::min(tnew, dtMax);
      *dt_io = std::max(tnew, dtMin);
      first = false;
    }
    q.p = int_params(c, used, c->Br, c->Bk);
    q.s = tb.nb - 1;
    q.last = tb.last_is_solution ? 1 : 0;
    for (int j = 0; j < 7; j++) q.a[j] = tb.b[j];
    c->launches += launch_rk_accept(c->stream, q, fp64(c));
    c->launches += launch_obs(c->stream, obs_params(c, used));
    t += used;
    done++;
  }
  CK(c, cudaGetLastError());
  c->have_geometry = true;
  if (steps_done) *steps_done = done;
  return read_err_word(c);
}

// ------------------------------------------------------------ checkpoints
// Binary snapshot of a context: "MDCKPT01", then int64 n, precision, kc,
// noise mode, seed, step; double box length, alpha, rc, time; rMag[n],
// rHydr[n]; pos, mm, ea, truePos, posRef as N x 3 column-major FP64.

namespace {
const char kCkptMagic[8] = {'M', 'D', 'C', 'K', 'P', 'T', '0', '1'};
}

int md_checkpoint_save(md_ctx* c, const char* path) {
  int st = check_ready(c, true);
  if (st) return st;
  if (!path) return set_err(c, MD_ERR_INVALID, "null path");
  CK(c, cudaStreamSynchronize(c->stream));
  const size_t n = (size_t)c->n, B = 24 * n;
  std::vector<double> arr(15 * n);
  double* dev[5] = {c->pos, c->mm, c->ea, c->truePos, c->posRef};
  for (int q = 0; q < 5; q++) CK(c, cudaMemcpy(arr.data() + 3 * n * q, dev[q], B, cudaMemcpyDeviceToHost));
  double t = 0;
  int64_t step = 0;
  if ((st = md_get_time(c, &t, &step))) return st;
  FILE* f = std::fopen(path, "wb");
  if (!f) return set_err(c, MD_ERR_INVALID, "cannot open %s for writing", path);
  const int64_t hi[6] = {c->n, c->prec, c->kc, c->noise, (int64_t)c->seed, step};
  const double hd[4] = {c->L, c->alpha, c->rc, t};
  bool ok = std::fwrite(kCkptMagic, 1, 8, f) == 8 && std::fwrite(hi, 8, 6, f) == 6 && std::fwrite(hd, 8, 4, f) == 4 &&
            std::fwrite(c->props.rMag.data(), 8, n, f) == n && std::fwrite(c->props.rHydr.data(), 8, n, f) == n &&
            std::fwrite(arr.data(), 8, 15 * n, f) == 15 * n;
  ok = (std::fclose(f) == 0) && ok;
  if (!ok) return set_err(c, MD_ERR_INVALID, "write to %s failed", path);
  // the saving run rebuilds its cell order and list at the next step, as a
  // run restored from this file does, so both continue identically
  return force_rebuild(c);
}

int md_checkpoint_load(md_ctx* c, const char* path) {
  if (!c || !path) return set_err(c, MD_ERR_INVALID, "null argument");
  FILE* f = std::fopen(path, "rb");
  if (!f) return set_err(c, MD_ERR_INVALID, "cannot open %s", path);
  char magic[8];
  int64_t hi[6];
  double hd[4];
  bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, kCkptMagic, 8) == 0 &&
            std::fread(hi, 8, 6, f) == 6 && std::fread(hd, 8, 4, f) == 4;
  if (!ok || hi[0] != c->n || hi[1] != c->prec) {
    std::fclose(f);
    return set_err(c, MD_ERR_INVALID, "%s is not a checkpoint of %lld particles in this precision", path,
                   (long long)c->n);
  }
  const size_t n = (size_t)c->n, B = 24 * n;
  std::vector<double> rMag(n), rHydr(n), arr(15 * n);
  ok = std::fread(rMag.data(), 8, n, f) == n && std::fread(rHydr.data(), 8, n, f) == n &&
       std::fread(arr.data(), 8, 15 * n, f) == 15 * n;
  std::fclose(f);
  if (!ok) return set_err(c, MD_ERR_INVALID, "%s is truncated", path);
  int st;
  if ((st = md_set_particles(c, rMag.data(), rHydr.data()))) return st;
  if ((st = md_set_box(c, hd[0]))) return st;
  if ((st = md_set_ewald(c, hd[1], hd[2], hi[2]))) return st;
  if ((st = md_state_upload(c, arr.data(), arr.data() + 3 * n, arr.data() + 6 * n, 0))) return st;
  CK(c, cudaMemcpy(c->truePos, arr.data() + 9 * n, B, cudaMemcpyHostToDevice));
  CK(c, cudaMemcpy(c->posRef, arr.data() + 12 * n, B, cudaMemcpyHostToDevice));
  if ((st = md_set_noise(c, (int)hi[3], (uint64_t)hi[4]))) return st;
  if ((st = md_set_time(c, hd[3], hi[5]))) return st;
  return force_rebuild(c);
}

int md_num_records(const md_ctx* cc, int64_t* count) {
  md_ctx* c = const_cast<md_ctx*>(cc);
  if (!c || !count) return MD_ERR_INVALID;
  long long n = 0;
  CK(c, cudaStreamSynchronize(c->stream));
  CK(c, cudaMemcpy(&n, &c->sc->nrec, sizeof n, cudaMemcpyDeviceToHost));
  *count = n;
  return MD_OK;
}

int md_records(md_ctx* c, int64_t first, int64_t count, double* obs) {
  int64_t n = 0;
  int st = md_num_records(c, &n);
  if (st) return st;
  if (first < 0 || count < 0 || first + count > n || (!obs && count)) return set_err(c, MD_ERR_INVALID, "bad record range");
  if (count) CK(c, cudaMemcpy(obs, c->records + 8 * first, 64 * (size_t)count, cudaMemcpyDeviceToHost));
  return MD_OK;
}

int md_clear_records(md_ctx* c) {
  if (!c) return MD_ERR_INVALID;
  CK(c, cudaMemsetAsync(&c->sc->nrec, 0, sizeof(long long), c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  c->nrec_bound = 0;
  return MD_OK;
}

int md_sync(md_ctx* c) {
  if (!c) return MD_ERR_INVALID;
  CK(c, cudaStreamSynchronize(c->stream));
  return MD_OK;
}

int md_debug_cells(md_ctx* c, int64_t* ncell, int64_t* ncx, int32_t* cell_start, int32_t* perm) {
  if (!c || !c->have_geometry) return set_err(c, MD_ERR_INVALID, "no cell list yet");
  CK(c, cudaStreamSynchronize(c->stream));
  if (ncell) *ncell = c->grid.ncell;
  if (ncx) *ncx = c->grid.ncx;
  if (cell_start) CK(c, cudaMemcpy(cell_start, c->cell_start, 4 * (size_t)(c->grid.ncell + 1), cudaMemcpyDeviceToHost));
  if (perm) CK(c, cudaMemcpy(perm, c->perm, 4 * (size_t)c->n, cudaMemcpyDeviceToHost));
  return MD_OK;
}

int md_debug_structure_factor(md_ctx* c, int64_t* nk_inout, double* out5) {
  if (!c || !nk_inout || !c->have_geometry) return set_err(c, MD_ERR_INVALID, "no structure factor yet");
  const int nk = c->klist.nk;
  std::vector<double2> S(nk);
  CK(c, cudaStreamSynchronize(c->stream));
  CK(c, cudaMemcpy(S.data(), c->Sfull, sizeof(double2) * nk, cudaMemcpyDeviceToHost));
  int64_t cnt = 0;
  for (int k = 0; k < nk; k++) {
    if (!c->klist.kreal[k]) continue;
    if (out5 && cnt < *nk_inout) {
      double* o = out5 + 5 * cnt;
      o[0] = c->klist.kx[k];
      o[1] = c->klist.ky[k];
      o[2] = c->klist.kz[k];
      o[3] = S[k].x * c->props.muMax;
      o[4] = S[k].y * c->props.muMax;
    }
    cnt++;
  }
  *nk_inout = cnt;
  return MD_OK;
}

int md_debug_launches(const md_ctx* c, int64_t* launches) {
  if (!c || !launches) return MD_ERR_INVALID;
  *launches = c->launches;
  return MD_OK;
}

int md_debug_pairs(md_ctx* c, int64_t* pairs) {
  if (!c || !pairs) return set_err(c, MD_ERR_INVALID, "null argument");
  if (int st = count_pairs(c)) return st;
  *pairs = c->pairs;
  return MD_OK;
}

int md_set_neighbor_skin(md_ctx* c, double skin_frac) {
  if (!c || !(skin_frac >= 0) || skin_frac > 1) return set_err(c, MD_ERR_INVALID, "skin fraction must be in [0, 1]");
  if (int st = count_pairs(c)) return st;
  c->skin_frac = skin_frac;
  c->cell_skin = std::max(c->cell_skin, skin_frac);
  c->list_valid = false;
  invalidate_graph(c);
  if (c->have_ewald) {
    const int64_t cap = mdh::list_entries(c->n, c->rc / c->L * (1.0 + c->skin_frac));
    if (int st = alloc_nbr(c, cap, true)) return st;
  }
  return force_rebuild(c);
}

int md_set_strong_pairs(md_ctx* c, double theta) {
  if (!c || !(theta >= 0)) return set_err(c, MD_ERR_INVALID, "strong-pair threshold must be >= 0 (0: off)");
  CK(c, cudaStreamSynchronize(c->stream));
  c->strong_theta = theta;
  invalidate_graph(c);
  if (!c->have_ewald) return MD_OK;
  update_strong(c);
  if (c->strong_w4sq > 0.f && !c->cfg.ENABLE_COATING_POT)
    if (int st = alloc_strong(c, strong_entries(c))) return st;
  return force_rebuild(c);
}

int md_debug_strong_pairs(md_ctx* c, int64_t* entries) {
  if (!c || !entries) return set_err(c, MD_ERR_INVALID, "null argument");
  *entries = 0;
  if (!strong_active(c)) return MD_OK;
  CK(c, cudaStreamSynchronize(c->stream));
  StepFlags f;
  int total = 0;
  CK(c, cudaMemcpy(&f, &c->sc->flags, sizeof f, cudaMemcpyDeviceToHost));
  CK(c, cudaMemcpy(&total, c->snbr_off + c->n, sizeof(int), cudaMemcpyDeviceToHost));
  *entries = (f.overflow || f.soverflow) ? -1 : total;
  return MD_OK;
}

int md_set_wait_limit(md_ctx* c, int64_t cycles) {
  if (!c || cycles < 1000) return set_err(c, MD_ERR_INVALID, "wait limit must be >= 1000 cycles");
  CK(c, cudaStreamSynchronize(c->stream));
  c->tc_wait = cycles;
  invalidate_graph(c);
  return MD_OK;
}

int md_debug_wait_probe(md_ctx* c, int arrive, int64_t cycles) {
  if (!c || cycles < 1000) return set_err(c, MD_ERR_INVALID, "wait limit must be >= 1000 cycles");
  launch_tc_wait_probe(c->stream, &c->sc->err, arrive ? 1 : 0, cycles);
  CK(c, cudaGetLastError());
  return read_err_word(c);
}

int md_debug_real_part(md_ctx* c, double* B, double* F) {
  if (!c || !B || !F) return set_err(c, MD_ERR_INVALID, "null argument");
  if (!c->have_geometry) return set_err(c, MD_ERR_INVALID, "call md_compute_interactions first");
  IntParams ip = int_params(c, 0.0, c->Br, c->Bk);
  launch_real_part(c->stream, ip, c->Bout, c->Fout, fp64(c));
  CK(c, cudaGetLastError());
  CK(c, cudaMemcpyAsync(B, c->Bout, 24 * (size_t)c->n, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaMemcpyAsync(F, c->Fout, 24 * (size_t)c->n, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  return MD_OK;
}

int md_debug_neighbor_capacity(md_ctx* c, int64_t cap, int64_t* used) {
  if (!c) return MD_ERR_INVALID;
  CK(c, cudaStreamSynchronize(c->stream));
  if (used) {
    int total = 0;
    CK(c, cudaMemcpy(&total, c->nbr_off + c->n, sizeof(int), cudaMemcpyDeviceToHost));
    *used = total;
  }
  if (cap > 0) {
    // shrink only the usable capacity; the allocation stays
    c->nbr_cap = std::min<long long>(cap, c->nbr_cap);
    invalidate_graph(c);
    return force_rebuild(c);
  }
  return MD_OK;
}

int md_profile(md_ctx* c, int enable) {
  if (!c) return MD_ERR_INVALID;
  if (enable && !c->ev[0])
    for (int k = 0; k <= MD_NSEG; k++) CK(c, cudaEventCreate(&c->ev[k]));
  if ((bool)enable != c->prof) invalidate_graph(c);
  c->prof = enable != 0;
  return MD_OK;
}

int md_profile_read(md_ctx* c, double* ms) {
  if (!c || !ms || !c->prof) return set_err(c, MD_ERR_INVALID, "profiling not enabled");
  CK(c, cudaStreamSynchronize(c->stream));
  for (int k = 0; k < MD_NSEG; k++) {
    float t = 0;
    CK(c, cudaEventElapsedTime(&t, c->ev[k], c->ev[k + 1]));
    ms[k] = t;
  }
  return MD_OK;
}

int md_calibrate_fp32(double* tflops) {
  if (!tflops) return set_err(nullptr, MD_ERR_INVALID, "null argument");
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return set_err(nullptr, MD_ERR_NO_DEVICE, "no CUDA device");
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int threads = 256, blocks = nsm * 8;
  float* out = nullptr;
  cudaStream_t st;
  cudaEvent_t e0, e1;
  CK(nullptr, cudaMalloc(&out, sizeof(float) * threads * blocks));
  CK(nullptr, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  CK(nullptr, cudaEventCreate(&e0));
  CK(nullptr, cudaEventCreate(&e1));
  double best = 0;
  for (int rep = 0; rep < 6; rep++) {
    cudaEventRecord(e0, st);
    double flops = 0;
    for (int q = 0; q < 4; q++) flops += launch_fma_calibration(st, out, blocks, threads);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && ms > 0) best = std::max(best, flops / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  cudaFree(out);
  *tflops = best;
  return best > 0 ? MD_OK : set_err(nullptr, MD_ERR_CUDA, "calibration failed");
}

// Timing of one candidate: the evaluations of a Heun step (field + force,
// then field only; the integrator's kernels are the same for every
// candidate), the median of kTuneReps repetitions after one that builds the
// lists, each after a write of a buffer larger than L2, as the steps of a
// run find the cache.
namespace {
constexpr int kTuneReps = 5;
// A candidate replaces the cost model's choice (or the default tiling) only
// when it is faster by more than this fraction: closer results are within
// the repetition-to-repetition spread.
constexpr double kTuneMargin = 0.03;
}  // namespace

static double time_evaluations(md_ctx* c, cudaEvent_t e0, cudaEvent_t e1, void* flush, size_t flush_bytes) {
  float t[kTuneReps];
  for (int rep = 0; rep <= kTuneReps; rep++) {
    if (flush) cudaMemsetAsync(flush, rep & 1, flush_bytes, c->stream);
    cudaEventRecord(e0, c->stream);
    issue_interactions(c);
    issue_field(c);
    cudaEventRecord(e1, c->stream);
    if (cudaEventSynchronize(e1) != cudaSuccess) return 1e300;
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0) t[rep - 1] = ms;
  }
  std::sort(t, t + kTuneReps);
  return t[kTuneReps / 2];
}

int md_autotune_ewald(md_ctx* c, int ncand, double* alpha_out, double* rc_out, int64_t* kc_out, double* best_ms) {
  int st = check_ready(c, false);
  if (!c || !c->have_particles) return set_err(c, MD_ERR_INVALID, "particles not set");
  if (!c->have_state) return set_err(c, MD_ERR_INVALID, "state not uploaded");
  (void)st;
  if (ncand < 1) ncand = 5;
  mdh::EwaldModel m = mdh::ewald_model(c->cfg, c->props);
  double a0;
  int64_t k0;
  const double rc0 = mdh::choose_rc(c->cfg, m, c->n, &a0, &k0, tc_kc_bound(c)) / c->L;
  cudaEvent_t e0, e1;
  CK(c, cudaEventCreate(&e0));
  CK(c, cudaEventCreate(&e1));
  // L2 flush buffer (twice the L2), freed at the end; without it the
  // candidates are timed on a warm cache
  int dev = 0, l2 = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
  const size_t flush_bytes = std::max<size_t>(2 * (size_t)std::max(l2, 0), 64u << 20);
  void* flush = nullptr;
  if (dalloc(c, &flush, flush_bytes) != MD_OK) {
    cudaGetLastError();
    flush = nullptr;
  }
  auto done = [&](int code) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    dfree(c, flush);
    return code;
  };
  // candidates: the cost model's cutoff first, then ncand cutoffs from
  // 0.75 to 1.35 times it
  std::vector<double> xs{rc0};
  if (ncand > 1)
    for (int q = 0; q < ncand; q++) xs.push_back(std::min(0.5, rc0 * (0.75 + 0.6 * q / (ncand - 1))));
  double best = 1e300, base = 1e300, ba = 0, brc = 0;
  int64_t bk = 0;
  for (size_t q = 0; q < xs.size(); q++) {
    const double x = xs[q];
    double a = a0, kr = (double)k0;  // q = 0: the cost model's (alpha, kc) as md_ewald_params gives them
    if (q > 0 && !mdh::ewald_for_rc(c->cfg, m, x * c->L, &a, &kr)) continue;
    const int64_t k = (int64_t)std::floor(kr + 0.5);
    if (k > 64 || md_set_ewald(c, a, x * c->L, k) != MD_OK) continue;
    const double ms = time_evaluations(c, e0, e1, flush, flush_bytes);
    if (q == 0) base = ms;
    // the first timed candidate (the cost model's) is the reference the
    // others must beat by the margin
    const bool better = best >= 1e300 || ms < best * (best == base ? 1.0 - kTuneMargin : 1.0);
    if (better) {
      best = ms;
      ba = a;
      brc = x * c->L;
      bk = k;
    }
  }
  if (best >= 1e300) return done(set_err(c, MD_ERR_INVALID, "no candidate cutoff met the error model"));
  if ((st = md_set_ewald(c, ba, brc, bk))) return done(st);
  // at the chosen cutoff: the k-space engine and, on the tensor cores, the
  // structure factor's ring option and chunk count (waves), timed the same
  // way; the default tiling first, kept unless beaten by the margin
  if (!fp64(c)) {
    struct Cand {
      int engine, ring, waves;
    };
    const int eng0 = c->kengine;
    std::vector<Cand> cands{{eng0, c->tc_ring, c->tc_waves}};
    if (md::kspace_tc_supported((int)bk) && eng0 != MD_KSPACE_SIMT) {
      int ro[6];
      const int nr = md::kspace_tc_ring_options((int)bk, ro, 6);
      for (int q = 0; q < nr && q < 3; q++)
        for (int w = 1; w <= 2; w++) cands.push_back({MD_KSPACE_AUTO, ro[q], w});
      cands.push_back({MD_KSPACE_SIMT, -1, 1});
    }
    double bms = 1e300, bms0 = 1e300;
    Cand bc = cands[0];
    for (size_t q = 0; q < cands.size(); q++) {
      const Cand& cd = cands[q];
      c->kengine = cd.engine;
      c->tc_ring = cd.ring;
      c->tc_waves = cd.waves;
      if (setup_engine(c) != MD_OK) continue;
      invalidate_graph(c);
      const double ms = time_evaluations(c, e0, e1, flush, flush_bytes);
      if (q == 0) bms0 = ms;
      if (bms >= 1e300 || ms < bms * (bms == bms0 ? 1.0 - kTuneMargin : 1.0)) {
        bms = ms;
        bc = cd;
      }
    }
    c->kengine = bc.engine;
    c->tc_ring = bc.ring;
    c->tc_waves = bc.waves;
    if ((st = setup_engine(c))) return done(st);
    invalidate_graph(c);
    c->have_geometry = false;
    if (bms < 1e300) best = std::min(best, bms);
  }
  done(MD_OK);
  if (alpha_out) *alpha_out = ba;
  if (rc_out) *rc_out = brc;
  if (kc_out) *kc_out = bk;
  if (best_ms) *best_ms = best;
  return MD_OK;
}

// Ewald cutoff cache per (N, volume fraction) bucket: N in half octaves,
// volume fraction in steps of 0.01.
namespace {
std::mutex g_tune_mu;
// bucket -> tuned choices: rc / L, k-space engine, structure-factor ring option, chunk waves
struct TuneEntry {
  double x;
  int engine, ring, waves;
};
std::map<std::pair<int, int>, TuneEntry> g_tune;
std::pair<int, int> tune_key(int64_t n, double volFrac) {
  return {(int)std::floor(2.0 * std::log2((double)n)), (int)std::lround(volFrac * 100.0)};
}
}  // namespace

int md_autotune_ewald_cached(md_ctx* c, double volFrac, double* alpha, double* rc, int64_t* kc, int* hit) {
  if (!c || !c->have_particles || !c->have_state) return set_err(c, MD_ERR_INVALID, "particles or state not set");
  const auto key = tune_key(c->n, volFrac);
  double x = -1;
  TuneEntry te{-1, MD_KSPACE_AUTO, -1, 1};
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find(key);
    if (it != g_tune.end()) te = it->second;
    x = te.x;
  }
  if (hit) *hit = x > 0;
  if (x > 0) {
    mdh::EwaldModel m = mdh::ewald_model(c->cfg, c->props);
    double a = 0, kr = 0;
    if (mdh::ewald_for_rc(c->cfg, m, x * c->L, &a, &kr)) {
      const int64_t k = std::max<int64_t>(1, (int64_t)std::floor(kr + 0.5));
      if (!fp64(c)) {
        c->kengine = te.engine;
        c->tc_ring = te.ring;
        c->tc_waves = te.waves;
      }
      int st = md_set_ewald(c, a, x * c->L, k);
      if (st == MD_OK) {
        if (alpha) *alpha = a;
        if (rc) *rc = x * c->L;
        if (kc) *kc = k;
        return MD_OK;
      }
    }
    if (hit) *hit = 0;  // the cached cutoff does not fit this system: tune it
  }
  double a = 0, r = 0;
  int64_t k = 0;
  int st = md_autotune_ewald(c, 5, &a, &r, &k, nullptr);
  if (st) return st;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[key] = TuneEntry{r / c->L, c->kengine, c->tc_ring, c->tc_waves};
  }
  if (alpha) *alpha = a;
  if (rc) *rc = r;
  if (kc) *kc = k;
  return MD_OK;
}

int md_tune_cache_save(const char* path) {
  if (!path) return set_err(nullptr, MD_ERR_INVALID, "null path");
  FILE* f = std::fopen(path, "w");
  if (!f) return set_err(nullptr, MD_ERR_INVALID, "cannot write %s", path);
  std::lock_guard<std::mutex> lk(g_tune_mu);
  std::fprintf(f, "# n_bucket(2*log2 N) volfrac_bucket(x100) rc_over_L kspace_engine sf_ring sf_waves\n");
  for (const auto& kv : g_tune)
    std::fprintf(f, "%d %d %.17g %d %d %d\n", kv.first.first, kv.first.second, kv.second.x, kv.second.engine,
                 kv.second.ring, kv.second.waves);
  std::fclose(f);
  return MD_OK;
}

int md_tune_cache_load(const char* path) {
  if (!path) return set_err(nullptr, MD_ERR_INVALID, "null path");
  FILE* f = std::fopen(path, "r");
  if (!f) return set_err(nullptr, MD_ERR_INVALID, "cannot read %s", path);
  char line[256];
  std::lock_guard<std::mutex> lk(g_tune_mu);
  while (std::fgets(line, sizeof line, f)) {
    int a = 0, b = 0, eng = MD_KSPACE_AUTO, ring = -1, waves = 1;
    double x = 0;
    const int got = line[0] == '#' ? 0 : std::sscanf(line, "%d %d %lf %d %d %d", &a, &b, &x, &eng, &ring, &waves);
    if (got >= 3 && x > 0 && x <= 0.5) {
      if (got < 6 || eng < MD_KSPACE_AUTO || eng > MD_KSPACE_TC || ring < -1 || ring > 5 || waves < 1 || waves > 4) {
        eng = MD_KSPACE_AUTO;  // a line with the cutoff only: default k-space choices
        ring = -1;
        waves = 1;
      }
      g_tune[{a, b}] = TuneEntry{x, eng, ring, waves};
    }
  }
  std::fclose(f);
  return MD_OK;
}

int md_tune_cache_clear(void) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune.clear();
  return MD_OK;
}

}  // extern "C"

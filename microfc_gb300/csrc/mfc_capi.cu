// C ABI of the GB300 MicroFC hot path (declared in include/mfc_gpu.h).
//
// Host side: validates the case like s_check_input_file
// (src/simulation/m_start_up.fpp:117-290), builds the grid ghost layers
// (m_start_up.fpp:517-655) and the grid-dependent WENO coefficients
// (src/simulation/m_weno.fpp:168-363) once, uploads them, and drives the
// fused stage kernels for the TVD RK schemes of m_time_steppers.fpp and the
// time loop of p_main.fpp.
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/mfc_gpu.h"
#include "mfc_grid.h"
#include "mfc_ic.h"
#include "mfc_launch.h"

namespace {

thread_local std::string g_err = "";

int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

#define MFC_CUDA(call)                                                                            \
  do {                                                                                            \
    cudaError_t e_ = (call);                                                                      \
    if (e_ != cudaSuccess) return fail(MFC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

std::once_flag g_reg_once;
std::vector<mfc::StageEntry> g_reg;

void build_registry() {
  std::call_once(g_reg_once, [] {
    mfc::register_stage_1d_fp64(g_reg);
    mfc::register_stage_1d_fp32(g_reg);
    mfc::register_stage_2d_fp64(g_reg);
    mfc::register_stage_2d_fp64fma(g_reg);
    mfc::register_stage_2d_fp32(g_reg);
    mfc::register_stage_3d_fp64(g_reg);
    mfc::register_stage_3d_fp32(g_reg);
    mfc::register_stage_visc_fp64(g_reg);
    mfc::register_stage_visc_fp32(g_reg);
    mfc::register_stage_char_fp64(g_reg);
  });
}

}  // namespace

namespace mfc {
const StageEntry* find_stage(int nd, int nf, int wo, int prec, bool visc, bool chr) {
  build_registry();
  for (const auto& e : g_reg)
    if (e.nd == nd && e.nf == nf && e.wo == wo && e.prec == prec && e.visc == visc && e.chr == chr) return &e;
  return nullptr;
}

int report_error(int code, const std::string& msg) { return fail(code, msg); }

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif
void populate_pages(void* p, size_t bytes) {
  if (!p || bytes == 0) return;
  static const size_t page = [] {
    const long s = sysconf(_SC_PAGESIZE);
    return s > 0 ? (size_t)s : (size_t)4096;
  }();
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {  // no device, or an earlier error that the copy will report
    (void)cudaGetLastError();
    return;
  }
  if (at.type != cudaMemoryTypeUnregistered && at.type != cudaMemoryTypeHost) return;
  volatile char* c = static_cast<volatile char*>(p);
  auto touch = [&](auto&& f) {
    for (size_t i = 0; i < bytes; i += page) f(c + i);
    f(c + bytes - 1);
  };
  const uintptr_t first = reinterpret_cast<uintptr_t>(p) / page * page;
  const size_t pages = (reinterpret_cast<uintptr_t>(p) + bytes - first + page - 1) / page;
  if (at.type == cudaMemoryTypeUnregistered && pages <= 256) {
    touch([](volatile char* x) { *x = 0; });
    return;
  }
  if (at.type == cudaMemoryTypeUnregistered) {
    unsigned char in[16];
    bool resident = mincore(reinterpret_cast<void*>(first + pages / 2 * page), sizeof(in) * page, in) == 0;
    for (unsigned char k : in) resident = resident && (k & 1);
    if (!resident) {
      (void)madvise(reinterpret_cast<void*>(first), pages * page, MADV_POPULATE_WRITE);
      return;
    }
  }
  touch([](volatile char* x) { (void)*x; });
}

namespace {
// the driver's encoder, looked up through the runtime (no link against libcuda)
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled tiled_encoder() {
  static const EncodeTiled encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return static_cast<EncodeTiled>(nullptr);
    return reinterpret_cast<EncodeTiled>(fn);
  }();
  return encode;
}

// FP64 (elem_bytes 8) or FP32 (4) tensor of `rank` dimensions (x first, the
// variable last); strides in elements for dimensions 1.. .  TMA rules:
// 16-byte aligned base and strides, boxes of at most 256 cells per
// dimension whose rows are a multiple of 16 bytes.
bool encode_tensor(TileMap& t, const void* base, int elem_bytes, int rank, const int64_t* dims,
                   const int64_t* strides, const int* box) {
  std::memset(&t, 0, sizeof(t));
  const EncodeTiled encode = tiled_encoder();
  if (!encode || !base || reinterpret_cast<uintptr_t>(base) % 16 != 0 || (elem_bytes != 8 && elem_bytes != 4))
    return false;
  cuuint64_t gd[5], gs[4];
  cuuint32_t bd[5], unit[5];
  for (int d = 0; d < rank; ++d) {
    if (dims[d] < 1 || box[d] < 1 || box[d] > 256) return false;
    gd[d] = cuuint64_t(dims[d]);
    bd[d] = cuuint32_t(box[d]);
    unit[d] = 1;
    if (d > 0) {
      if ((strides[d - 1] * elem_bytes) % 16 != 0 || strides[d - 1] * elem_bytes >= (int64_t(1) << 40)) return false;
      gs[d - 1] = cuuint64_t(strides[d - 1]) * elem_bytes;
    }
  }
  if ((box[0] * elem_bytes) % 16 != 0) return false;
  const CUresult r =
      encode(&t.map, elem_bytes == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
             cuuint32_t(rank), const_cast<void*>(base), gd, gs, bd, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    std::memset(&t, 0, sizeof(t));
    return false;
  }
  t.on = 1;
  return true;
}
}  // namespace

bool encode_tile_map(TileMap& t, const double* base, int nx, int ny, int S, int64_t sy, int64_t sv, int box_w,
                     int box_h) {
  if (sy < nx || sv < sy * ny) {
    std::memset(&t, 0, sizeof(t));
    return false;
  }
  const int64_t dims[3] = {nx, ny, S}, strides[2] = {sy, sv};
  const int box[3] = {box_w, box_h, S};
  return encode_tensor(t, base, 8, 3, dims, strides, box);
}

bool encode_tile_map_3d(TileMap& t, const void* base, int elem_bytes, int nx, int ny, int nz, int S, int64_t sy,
                        int64_t sz, int64_t sv, int bx, int by, int bz) {
  if (sy < nx || sz < sy * ny || sv < sz * nz) {
    std::memset(&t, 0, sizeof(t));
    return false;
  }
  const int64_t dims[4] = {nx, ny, nz, S}, strides[3] = {sy, sz, sv};
  const int box[4] = {bx, by, bz, S};
  return encode_tensor(t, base, elem_bytes, 4, dims, strides, box);
}
}  // namespace mfc

struct mfc_gpu_ctx {
  mfc_params prm{};
  int nd = 1, S = 0, b = 0;
  int n[3] = {1, 1, 1};
  int64_t pitch = 0, sy = 0, sz = 0, sv = 0, reg_elems = 0;
  double* state = nullptr;      // 3 registers
  double* reg[3] = {nullptr, nullptr, nullptr};
  double* rhs = nullptr;
  double* work = nullptr;       // 3-D: partial RHS between the directional sweeps, then the primitives
  void* gate_w = nullptr;       // MFC_PREC_GATED: FP16 gate parameters
  uint8_t* gate_flags = nullptr;  // MFC_PREC_GATED: a step's first-stage gate decisions
  bool gate_ready = false;
  // split and gated 2-D (null where there was no room) and split 3-D WENO5:
  // the primitive pairs of the last stage's output (prim[prim_at]; of register
  // prim_of, or of none), and the buffer that the next stage writes them to
  mfc::f32x2* prim[2] = {nullptr, nullptr};
  int prim_at = 0;
  const double* prim_of = nullptr;
  bool captured = false;  // a graph holds launches of this context: its replays change registers and pairs unseen
  unsigned long long* monitor = nullptr;  // max ICFL of the monitored steps (double bits)
  bool monitor_on = false;
  double* tables = nullptr;     // inv_d and coefficient tables
  uint32_t* status = nullptr;
  cudaStream_t stream = nullptr;
  // asynchronous snapshots: per slot a device staging copy and a pinned host buffer
  double* snap_dev[2] = {nullptr, nullptr};
  double* snap_host[2] = {nullptr, nullptr};
  cudaStream_t copy_stream = nullptr;
  // viscous parameters as uploaded (host copy), and weno_Re_flux = T's
  // gradient preparation
  mfc::ViscParams visc_host{};
  bool wrf = false;
  mfc::ViscGradBuffers vg;
  // device scratch of the standalone WENO / Riemann entry points, kept
  // between calls and grown to the largest request
  void* scratch = nullptr;
  size_t scratch_bytes = 0;
  cudaEvent_t snap_staged = nullptr, snap_done[2] = {nullptr, nullptr};
  bool snap_pending[2] = {false, false};
  // processor boundaries: receive buffers per side ([2*dir + side]) and their device table
  bool has_proc = false;
  int H = 0;
  double* halo_buf[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  int64_t halo_count[6] = {0, 0, 0, 0, 0, 0};
  const double** halo_table = nullptr;
  std::vector<double> cb_host[3];      // the cell boundaries passed at init
  std::vector<double> ghost_w[3][2];   // neighbour widths of processor boundaries
  mfc::ViscParams* visc = nullptr;     // device copy (viscous cases)
  bool chr = false;                    // WENO of the characteristic fields
  size_t off_dcc[3] = {0, 0, 0};       // spacing tables inside `tables`
  mfc::DevParams dev{};
  mfc::UniformCoef ucoef{};        // uniform grids: the split kernels' shared coefficient records
  mfc::UniformCoef ucoef_found{};  // what the grid tables allow
  bool ucoef_enabled = true;       // ucoef = ucoef_found when enabled, else all off
  const mfc::StageEntry* stage = nullptr;
  int64_t launches = 0;
};

namespace mfc {
bool ctx_view(mfc_gpu_ctx* c, CtxView& v) {
  if (!c) return false;
  v.dev = &c->dev;
  v.q0 = c->reg[0];
  v.stream = c->stream;
  v.nd = c->nd;
  v.nf = c->prm.num_fluids;
  v.wo = c->prm.weno_order;
  v.S = c->S;
  v.prec = c->prm.precision;
  for (int d = 0; d < 3; ++d) v.n[d] = c->n[d];
  v.visc = c->visc != nullptr;
  v.has_proc = c->has_proc;
  v.launches = &c->launches;
  return true;
}

cudaError_t ctx_scratch(mfc_gpu_ctx* c, size_t bytes, void** out) {
  if (bytes > c->scratch_bytes) {
    // the entry points that use it synchronise before they return, so the
    // old buffer is idle
    cudaFree(c->scratch);
    c->scratch = nullptr;
    c->scratch_bytes = 0;
    const cudaError_t e = cudaMalloc(&c->scratch, bytes);
    if (e != cudaSuccess) return e;
    c->scratch_bytes = bytes;
  }
  *out = c->scratch;
  return cudaSuccess;
}
}  // namespace mfc

namespace {

int validate(const mfc_params* p) {
  const std::string why = mfc::validate_params(p, /*allow_processor=*/true);
  return why.empty() ? MFC_OK : fail(MFC_ERR_INVALID, why);
}

// cudaMalloc for the buffers that come after mfc_gpu_init: where it finds no
// room, a 2-D context gives its primitive pairs back first (not those that a
// captured graph points to).
template <class T>
cudaError_t ctx_malloc(mfc_gpu_ctx* c, T** ptr, size_t bytes) {
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e == cudaErrorMemoryAllocation && c->nd == 2 && c->prim[0] != nullptr && !c->captured) {
    (void)cudaGetLastError();
    if ((e = cudaStreamSynchronize(c->stream)) != cudaSuccess) return e;
    cudaFree(c->prim[0]);
    c->prim[0] = c->prim[1] = nullptr;
    c->prim_of = nullptr;
    e = cudaMalloc(ptr, bytes);
  }
  return e;
}

// follows: qin is what this call's previous launch made
int launch_stage(mfc_gpu_ctx* c, const double* qin, const double* qbase, double* qout, double dt, int kind,
                 bool last_stage = false, bool follows = false) {
  mfc::DevParams P = c->dev;
  if (last_stage && c->monitor_on) P.monitor = c->monitor;  // ICFL of the step's new state
  if (c->wrf && c->visc) {  // weno_Re_flux = T: the stage input's face gradients first
    const bool fp32 = c->prm.precision != MFC_PREC_FP64;  // split or gated (contracted FP64 is refused)
    const cudaError_t g = mfc::visc_gradients_launch(c->nd, c->prm.num_fluids, fp32, c->dev, c->vg, qin, c->stream);
    if (g != cudaSuccess) return fail(MFC_ERR_CUDA, std::string("viscous gradients: ") + cudaGetErrorString(g));
    c->launches += mfc::visc_gradients_launches(c->nd, fp32);
  }
  cudaError_t e;
  if (c->prim[0] != nullptr && c->stage->launch_prims != nullptr) {
    const bool keep = kind != mfc::kRhsOnly;  // an RHS evaluation makes no state
    const int64_t pitch = mfc::prim_pitch(c->n[0]);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(c->stream, &capture);
    if (e != cudaSuccess) return fail(MFC_ERR_CUDA, std::string("stage launch: ") + cudaGetErrorString(e));
    c->captured |= capture != cudaStreamCaptureStatusNone;
    // 3-D stages always have the pairs of their input somewhere: an RHS
    // evaluation's go where they spare the last stage's
    const bool have = c->prim_of == qin && (follows || !c->captured);
    const mfc::PrimPairs B{have ? c->prim[c->prim_at] : nullptr, keep ? c->prim[c->prim_at ^ 1] : nullptr, pitch,
                           pitch * c->n[1], c->prim[have || keep ? c->prim_at : c->prim_at ^ 1]};
    e = c->stage->launch_prims(P, c->ucoef, qin, qbase, qout, dt, kind, B, c->stream);
    if (keep) {
      c->prim_at ^= 1;
      c->prim_of = e == cudaSuccess ? qout : nullptr;
    }
  } else {
    e = c->stage->launch(P, c->ucoef, qin, qbase, qout, dt, kind, c->stream);
    if (kind != mfc::kRhsOnly) c->prim_of = nullptr;  // the registers change, the pairs do not
  }
  if (e != cudaSuccess) return fail(MFC_ERR_CUDA, std::string("stage launch: ") + cudaGetErrorString(e));
  c->launches += c->stage->kernels;
  return MFC_OK;
}

// cons -> prim of the interior cells (for mfc_gpu_compute_rhs's prim output).
template <int ND, int NF>
__global__ void prim_kernel(const mfc::DevParams P, const double* __restrict__ q, double* __restrict__ out) {
  using Q = mfc::Eqs<ND, NF>;
  const int64_t cells = (int64_t)P.n[0] * P.n[1] * P.n[2];
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < cells; c += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(c % P.n[0]);
    const int y = (int)((c / P.n[0]) % P.n[1]);
    const int z = (int)(c / ((int64_t)P.n[0] * P.n[1]));
    const int64_t o = z * P.sz + y * P.sy + x;
    double v[Q::S];
#pragma unroll
    for (int k = 0; k < Q::S; ++k) v[k] = q[o + k * P.sv];
    mfc::cons_to_prim<ND, NF>(v, P);
#pragma unroll
    for (int k = 0; k < Q::S; ++k) out[o + k * P.sv] = v[k];
  }
}

// Boundary strip of a stage input for the neighbour across (dir, side), in
// the neighbour's halo layout (depth d = 0 is the cell next to the
// boundary): dir 0 [S][nz][ny][H], dir 1 [S][nz][H][nx], dir 2 [S][H][ny][nx].
// Strip of one processor boundary for the neighbour's receive buffer.  In
// 2-D the y strips are widened by one column on each side (wy = nx + 2): the
// x ghost cells -1 and nx of the packed rows, taken from this subdomain's own
// x receive buffers (xh0/xh1, depth 0) where x is a processor boundary, else
// from its x boundary condition.  They carry the diagonal neighbour's cells
// to the y neighbour, whose viscous corner gradients read them; the x
// strips must therefore have arrived before the y strips are packed.
__global__ void halo_pack_kernel(const double* __restrict__ q, int S, int nx, int ny, int nz, int64_t sy, int64_t sz,
                                 int64_t sv, int H, int dir, int side, int wy, const double* __restrict__ xh0,
                                 const double* __restrict__ xh1, int bcx_beg, int bcx_end, int mom,
                                 double* __restrict__ dst) {
  const int64_t total = (int64_t)S * H * (dir == 0 ? (int64_t)ny * nz : dir == 1 ? (int64_t)wy * nz : (int64_t)nx * ny);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, z, d, v;
    if (dir == 0) {
      d = (int)(i % H);
      y = (int)((i / H) % ny);
      z = (int)((i / ((int64_t)H * ny)) % nz);
      v = (int)(i / ((int64_t)H * ny * nz));
      x = side == 0 ? d : nx - 1 - d;
    } else if (dir == 1) {
      x = (int)(i % wy) - (wy - nx) / 2;
      d = (int)((i / wy) % H);
      z = (int)((i / ((int64_t)wy * H)) % nz);
      v = (int)(i / ((int64_t)wy * H * nz));
      y = side == 0 ? d : ny - 1 - d;
      if (x < 0 || x >= nx) {  // widened 2-D strip: an x ghost cell of row y
        const double* xh = x < 0 ? xh0 : xh1;
        if (xh) {
          dst[i] = xh[(int64_t)(v * ny + y) * H];
        } else {
          bool flip = false;
          const int gx = mfc::map_cell(x, nx, bcx_beg, bcx_end, &flip);
          const double val = q[v * sv + y * sy + gx];
          dst[i] = (flip && v == mom) ? -val : val;
        }
        continue;
      }
    } else {
      x = (int)(i % nx);
      y = (int)((i / nx) % ny);
      d = (int)((i / ((int64_t)nx * ny)) % H);
      v = (int)(i / ((int64_t)nx * ny * H));
      z = side == 0 ? d : nz - 1 - d;
    }
    dst[i] = q[v * sv + z * sz + y * sy + x];
  }
}

// Elements of the strip across direction dir (2-D y strips are widened by
// the two x ghost cells).
int64_t strip_elems(const mfc_gpu_ctx* c, int dir) {
  const int64_t wy = c->nd == 2 ? c->n[0] + 2 : c->n[0];
  return (int64_t)c->S * c->H *
         (dir == 0 ? (int64_t)c->n[1] * c->n[2] : dir == 1 ? wy * c->n[2] : (int64_t)c->n[0] * c->n[1]);
}

int copy_var(mfc_gpu_ctx* c, double* dev_reg, int var, const double* host, double* host_out, int64_t ld_y,
             int64_t ld_z) {
  if (var < 0 || var >= c->S) return fail(MFC_ERR_INVALID, "variable index out of range");
  if (ld_y < c->n[0] || (c->n[2] > 1 && ld_z < ld_y * c->n[1]))
    return fail(MFC_ERR_INVALID, "leading dimension smaller than the interior extent");
  for (int z = 0; z < c->n[2]; ++z) {
    double* d = dev_reg + var * c->sv + z * c->sz;
    if (host) {
      MFC_CUDA(cudaMemcpy2DAsync(d, (size_t)c->sy * 8, host + z * ld_z, (size_t)ld_y * 8, (size_t)c->n[0] * 8,
                                 (size_t)c->n[1], cudaMemcpyHostToDevice, c->stream));
    } else {
      MFC_CUDA(cudaMemcpy2DAsync(host_out + z * ld_z, (size_t)ld_y * 8, d, (size_t)c->sy * 8, (size_t)c->n[0] * 8,
                                 (size_t)c->n[1], cudaMemcpyDeviceToHost, c->stream));
    }
  }
  return MFC_OK;
}

}  // namespace

extern "C" {

int mfc_gpu_abi_version(void) { return MFC_GPU_ABI_VERSION; }

const char* mfc_gpu_last_error(void) { return g_err.c_str(); }

int mfc_gpu_init(const mfc_params* p, mfc_gpu_ctx** out) {
  if (!out) return fail(MFC_ERR_INVALID, "ctx_out is NULL");
  *out = nullptr;
  int rc = validate(p);
  if (rc) return rc;
  build_registry();
  MFC_CUDA(cudaSetDevice(p->device));

  auto* c = new mfc_gpu_ctx();
  c->prm = *p;
  c->nd = 1 + (p->n > 0) + (p->p > 0);
  c->S = 2 * p->num_fluids + c->nd + 1;
  const int polyn = (p->weno_order - 1) / 2;
  c->b = polyn + 2;
  c->n[0] = p->m + 1;
  c->n[1] = p->n + 1;
  c->n[2] = p->p + 1;
  c->pitch = (c->n[0] + 31) / 32 * 32;  // 256-byte rows
  c->sy = c->pitch;
  c->sz = c->sy * c->n[1];
  c->sv = c->sz * c->n[2];
  c->reg_elems = c->sv * c->S;

  c->stage = mfc::find_stage(c->nd, p->num_fluids, p->weno_order, p->precision);
  if (!c->stage) {
    delete c;
    return fail(MFC_ERR_INVALID, "no kernel compiled for this dimensionality / fluid count / WENO order / precision");
  }

  auto cleanup = [&](int code) {
    mfc_gpu_finalize(c);
    return code;
  };
  cudaError_t e;
  if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_CUDA, cudaGetErrorString(e)));
  if ((e = cudaMalloc(&c->state, sizeof(double) * c->reg_elems * 3)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  if ((e = cudaMalloc(&c->rhs, sizeof(double) * c->reg_elems)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  if (p->precision == MFC_PREC_GATED && (e = cudaMalloc(&c->gate_w, mfc::kGateBufferBytes)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  if (p->precision == MFC_PREC_GATED &&
      (e = cudaMalloc(&c->gate_flags, mfc::gate_flag_bytes(c->n[0], c->n[1]))) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  // 3-D: the partial RHS, then the primitives the x sweep stores (S x sv
  // values each, in the reconstruction type: FP64 at most); split WENO5: three
  // quarters of it, for the partial RHS and two buffers of primitive pairs
  if (c->nd == 3 && (e = cudaMalloc(&c->work, sizeof(double) * c->reg_elems * 2)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  if (c->nd == 3 && p->weno_order == 5 && p->precision == MFC_PREC_SPLIT)
    for (int k = 0; k < 2; ++k) c->prim[k] = reinterpret_cast<mfc::f32x2*>(c->work) + (k + 1) * (c->reg_elems / 2);
  if ((e = cudaMalloc(&c->monitor, sizeof(unsigned long long))) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  cudaMemsetAsync(c->monitor, 0, sizeof(unsigned long long), c->stream);
  if ((e = cudaMalloc(&c->status, sizeof(uint32_t))) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  cudaMemsetAsync(c->state, 0, sizeof(double) * c->reg_elems * 3, c->stream);
  cudaMemsetAsync(c->status, 0, sizeof(uint32_t), c->stream);
  for (int r = 0; r < 3; ++r) c->reg[r] = c->state + r * c->reg_elems;

  // grid tables: per direction inv_d[n] then kNumCoef * (n + 2*pad) coefficients
  const int bcb[3] = {p->bc_x_beg, p->bc_y_beg, p->bc_z_beg};
  const int bce[3] = {p->bc_x_end, p->bc_y_end, p->bc_z_end};
  mfc::GridTables gt;
  const std::string why = mfc::build_grid_tables(p, c->nd, c->n, c->b, gt);
  if (!why.empty()) return cleanup(fail(MFC_ERR_INVALID, why));
  const std::vector<double>& host = gt.host;
  if ((e = cudaMalloc(&c->tables, sizeof(double) * host.size())) != cudaSuccess)
    return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
  if ((e = cudaMemcpy(c->tables, host.data(), sizeof(double) * host.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
    return cleanup(fail(MFC_ERR_CUDA, cudaGetErrorString(e)));

  {
    const double* cbs[3] = {p->x_cb, p->y_cb, p->z_cb};
    for (int d = 0; d < c->nd; ++d) c->cb_host[d].assign(cbs[d], cbs[d] + c->n[d] + 1);
  }
  // halo receive buffers of the processor boundaries
  c->H = (p->weno_order + 1) / 2;
  for (int d = 0; d < c->nd; ++d) {
    for (int side = 0; side < 2; ++side) {
      if ((side == 0 ? bcb[d] : bce[d]) < 0) continue;
      c->has_proc = true;
      const int k = 2 * d + side;
      c->halo_count[k] = strip_elems(c, d);
      if ((e = cudaMalloc(&c->halo_buf[k], sizeof(double) * c->halo_count[k])) != cudaSuccess)
        return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
      cudaMemsetAsync(c->halo_buf[k], 0, sizeof(double) * c->halo_count[k], c->stream);
    }
  }
  if (c->has_proc) {
    if ((e = cudaMalloc(&c->halo_table, sizeof(double*) * 6)) != cudaSuccess)
      return cleanup(fail(MFC_ERR_NOMEM, cudaGetErrorString(e)));
    if ((e = cudaMemcpy(c->halo_table, c->halo_buf, sizeof(double*) * 6, cudaMemcpyHostToDevice)) != cudaSuccess)
      return cleanup(fail(MFC_ERR_CUDA, cudaGetErrorString(e)));
  }

  for (int d = 0; d < 3; ++d) c->off_dcc[d] = gt.off_dcc[d];
  mfc::DevParams& D = c->dev;
  D.halo = c->halo_table;
  for (int d = 0; d < 3; ++d) {
    D.n[d] = c->n[d];
    D.bc_beg[d] = bcb[d];
    D.bc_end[d] = bce[d];
    D.inv_d[d] = d < c->nd ? c->tables + gt.off_inv[d] : nullptr;
    D.coef[d] = d < c->nd ? c->tables + gt.off_coef[d] : nullptr;
    D.cstride[d] = gt.cstride[d];
  }
  D.sy = c->sy;
  D.sz = c->sz;
  D.sv = c->sv;
  for (int f = 0; f < mfc::kMaxFluids; ++f) {
    D.gammas[f] = f < p->num_fluids ? p->gammas[f] : 0.0;
    D.pi_infs[f] = f < p->num_fluids ? p->pi_infs[f] : 0.0;
  }
  D.weno_eps = p->weno_eps;
  mfc::set_fp32_constants(D);
  mfc::uniform_records(gt, c->nd, c->n, p->weno_order, p->precision, c->ucoef_found);
  c->ucoef = c->ucoef_found;
  D.coff = mfc::kCoefPad;
  D.status = c->status;
  D.work = c->work;  // shares its slot with gate_flags: set the one in use
  if (c->gate_flags) D.gate_flags = c->gate_flags;
  D.gate_w = c->gate_w;

  // 2-D split and gated: two buffers of primitive pairs, the next stage's
  // input and output (not with processor boundaries, whose ghost cells come
  // as conservative values).  The last allocation, and not a needed one: a
  // state that leaves no room for them runs without (ctx_malloc gives them
  // back to a later allocation that needs the room).
  if (c->nd == 2 && p->weno_order == 5 && (p->precision == MFC_PREC_SPLIT || p->precision == MFC_PREC_GATED) &&
      !c->has_proc) {
    const size_t pairs = (size_t)((c->S + 1) / 2) * c->n[1] * mfc::prim_pitch(c->n[0]);
    if (cudaMalloc(&c->prim[0], 2 * sizeof(mfc::f32x2) * pairs) == cudaSuccess) c->prim[1] = c->prim[0] + pairs;
    else (void)cudaGetLastError();
  }

  if ((e = c->stage->prepare()) != cudaSuccess) return cleanup(fail(MFC_ERR_CUDA, cudaGetErrorString(e)));
  if ((e = cudaStreamSynchronize(c->stream)) != cudaSuccess) return cleanup(fail(MFC_ERR_CUDA, cudaGetErrorString(e)));
  *out = c;
  return MFC_OK;
}

int mfc_gpu_sys_size(const mfc_gpu_ctx* c) { return c ? c->S : 0; }

int mfc_gpu_upload(mfc_gpu_ctx* c, int var, const double* host_sf, int64_t ld_y, int64_t ld_z) {
  if (!c || !host_sf) return fail(MFC_ERR_INVALID, "NULL argument");
  c->prim_of = nullptr;
  int rc = copy_var(c, c->reg[0], var, host_sf, nullptr, ld_y, ld_z);
  if (rc) return rc;
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_download(mfc_gpu_ctx* c, int var, double* host_sf, int64_t ld_y, int64_t ld_z) {
  if (!c || !host_sf) return fail(MFC_ERR_INVALID, "NULL argument");
  int rc = copy_var(c, c->reg[0], var, nullptr, host_sf, ld_y, ld_z);
  if (rc) return rc;
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

// The whole state in one strided copy: every row of every variable is n[0]
// values, rows follow each other every n[0] values on the host and every
// sy (= the padded pitch) in the register, across variables too (sv = sy *
// rows per variable).
// rows of n[0] values that need no padding (a pitch of n[0]): the register is
// one contiguous block like the host array, and one linear copy moves it
int mfc_gpu_upload_state(mfc_gpu_ctx* c, const double* host_q) {
  if (!c || !host_q) return fail(MFC_ERR_INVALID, "NULL argument");
  c->prim_of = nullptr;
  const size_t rows = (size_t)c->S * c->n[1] * c->n[2];
  if (c->sy == c->n[0])
    MFC_CUDA(cudaMemcpyAsync(c->reg[0], host_q, rows * c->n[0] * 8, cudaMemcpyHostToDevice, c->stream));
  else
    MFC_CUDA(cudaMemcpy2DAsync(c->reg[0], (size_t)c->sy * 8, host_q, (size_t)c->n[0] * 8, (size_t)c->n[0] * 8, rows,
                               cudaMemcpyHostToDevice, c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_generate_ic(mfc_gpu_ctx* c, const mfc_patch* patches, int num_patches, const double* domain) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  c->prim_of = nullptr;
  mfc::IcTarget t{c->nd,
                  c->prm.num_fluids,
                  {c->n[0], c->n[1], c->n[2]},
                  c->sy,
                  c->sz,
                  c->sv,
                  c->prm.gammas,
                  c->prm.pi_infs,
                  c->reg[0],
                  {c->cb_host[0].data(), c->nd > 1 ? c->cb_host[1].data() : nullptr,
                   c->nd > 2 ? c->cb_host[2].data() : nullptr}};
  const std::string why = mfc::generate_ic(t, patches, num_patches, domain, c->stream, &c->launches);
  if (!why.empty()) return fail(MFC_ERR_INVALID, why);
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_download_state(mfc_gpu_ctx* c, double* host_q) {
  if (!c || !host_q) return fail(MFC_ERR_INVALID, "NULL argument");
  const size_t rows = (size_t)c->S * c->n[1] * c->n[2];
  mfc::populate_pages(host_q, rows * c->n[0] * 8);
  if (c->sy == c->n[0])
    MFC_CUDA(cudaMemcpyAsync(host_q, c->reg[0], rows * c->n[0] * 8, cudaMemcpyDeviceToHost, c->stream));
  else
    MFC_CUDA(cudaMemcpy2DAsync(host_q, (size_t)c->n[0] * 8, c->reg[0], (size_t)c->sy * 8, (size_t)c->n[0] * 8, rows,
                               cudaMemcpyDeviceToHost, c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_set_gate(mfc_gpu_ctx* c, const float* host_params) {
  if (!c || !host_params) return fail(MFC_ERR_INVALID, "NULL argument");
  if (!c->gate_w) return fail(MFC_ERR_INVALID, "the context was not created with MFC_PREC_GATED");
  int rc = mfc::gate_upload(host_params, c->gate_w, c->stream);
  if (rc) return rc;
  c->gate_ready = true;
  return MFC_OK;
}

int mfc_gpu_gate_samples(mfc_gpu_ctx* c, int dir, float* x_dev, float* dev_dev) {
  if (!c || !x_dev || !dev_dev) return fail(MFC_ERR_INVALID, "NULL argument");
  if (c->nd != 2 || dir < 0 || dir > 1) return fail(MFC_ERR_INVALID, "gate samples are taken from 2-D cases, dir 0 or 1");
  if (c->prm.weno_order != 5) return fail(MFC_ERR_INVALID, "gate samples need WENO5 coefficients");
  return mfc::gate_samples(c->dev, c->prm.num_fluids, c->reg[0], dir, x_dev, dev_dev, c->stream);
}

int mfc_gpu_compute_rhs(mfc_gpu_ctx* c, double* rhs_out, double* prim_out) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (c->gate_w && !c->gate_ready) return fail(MFC_ERR_INVALID, "gate parameters not set (mfc_gpu_set_gate)");
  int rc = launch_stage(c, c->reg[0], c->reg[0], c->rhs, 0.0, mfc::kRhsOnly);
  if (rc) return rc;
  const int64_t cells = (int64_t)c->n[0] * c->n[1] * c->n[2];
  mfc::populate_pages(rhs_out, (size_t)c->S * cells * 8);
  mfc::populate_pages(prim_out, (size_t)c->S * cells * 8);
  if (rhs_out) {
    for (int v = 0; v < c->S; ++v)
      if ((rc = copy_var(c, c->rhs, v, nullptr, rhs_out + v * cells, c->n[0], (int64_t)c->n[0] * c->n[1]))) return rc;
  }
  if (prim_out) {
    double* tmp = c->reg[2];  // scratch register; not live between time steps
    const int nf = c->prm.num_fluids;
    const unsigned blocks = (unsigned)std::min<int64_t>((cells + 255) / 256, 4096);
    if (c->nd == 1 && nf == 1) prim_kernel<1, 1><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    else if (c->nd == 1 && nf == 2) prim_kernel<1, 2><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    else if (c->nd == 2 && nf == 1) prim_kernel<2, 1><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    else if (c->nd == 2) prim_kernel<2, 2><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    else if (nf == 1) prim_kernel<3, 1><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    else prim_kernel<3, 2><<<blocks, 256, 0, c->stream>>>(c->dev, c->reg[0], tmp);
    MFC_CUDA(cudaGetLastError());
    c->launches += 1;
    for (int v = 0; v < c->S; ++v)
      if ((rc = copy_var(c, tmp, v, nullptr, prim_out + v * cells, c->n[0], (int64_t)c->n[0] * c->n[1]))) return rc;
  }
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_tvd_rk(mfc_gpu_ctx* c, double dt, int last_step) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (c->has_proc)
    return fail(MFC_ERR_INVALID, "processor boundaries: step with mfc_gpu_rk_stage and a halo exchange per stage");
  if (c->gate_w && !c->gate_ready) return fail(MFC_ERR_INVALID, "gate parameters not set (mfc_gpu_set_gate)");
  if (last_step) return MFC_OK;  // s_compute_rhs returns before any update at t_step_stop
  int rc;
  double** R = c->reg;
  switch (c->prm.time_stepper) {
    case 1:
      if ((rc = launch_stage(c, R[0], R[0], R[1], dt, mfc::kRkEuler, true))) return rc;
      std::swap(R[0], R[1]);
      return MFC_OK;
    case 2:
      if ((rc = launch_stage(c, R[0], R[0], R[1], dt, mfc::kRkEuler))) return rc;
      return launch_stage(c, R[1], R[0], R[0], dt, mfc::kRk2Final, true, true);
    default:
      if ((rc = launch_stage(c, R[0], R[0], R[1], dt, mfc::kRkEuler))) return rc;
      if ((rc = launch_stage(c, R[1], R[0], R[2], dt, mfc::kRk3Mid, false, true))) return rc;
      return launch_stage(c, R[2], R[0], R[0], dt, mfc::kRk3Final, true, true);
  }
}

int mfc_gpu_rk_stage(mfc_gpu_ctx* c, int stage, double dt) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (c->gate_w && !c->gate_ready) return fail(MFC_ERR_INVALID, "gate parameters not set (mfc_gpu_set_gate)");
  const int ts = c->prm.time_stepper;
  if (stage < 0 || stage >= ts) return fail(MFC_ERR_INVALID, "stage out of range for the time stepper");
  double** R = c->reg;
  const bool last = stage == ts - 1;
  if (ts == 1) {
    int rc = launch_stage(c, R[0], R[0], R[1], dt, mfc::kRkEuler, true);
    if (!rc) std::swap(R[0], R[1]);
    return rc;
  }
  if (stage == 0) return launch_stage(c, R[0], R[0], R[1], dt, mfc::kRkEuler);
  if (ts == 2) return launch_stage(c, R[1], R[0], R[0], dt, mfc::kRk2Final, true);
  if (stage == 1) return launch_stage(c, R[1], R[0], R[2], dt, mfc::kRk3Mid);
  return launch_stage(c, R[2], R[0], R[0], dt, mfc::kRk3Final, last);
}

int mfc_gpu_halo_buffer(mfc_gpu_ctx* c, int dir, int side, double** dev_ptr, int64_t* count) {
  if (!c || !dev_ptr || dir < 0 || dir > 2 || side < 0 || side > 1) return fail(MFC_ERR_INVALID, "bad halo side");
  *dev_ptr = c->halo_buf[2 * dir + side];
  if (count) *count = c->halo_count[2 * dir + side];
  if (!*dev_ptr) return fail(MFC_ERR_INVALID, "that side is not a processor boundary");
  return MFC_OK;
}

int mfc_gpu_set_halo_widths(mfc_gpu_ctx* c, int dir, int side, const double* widths, int count) {
  if (!c || !widths || dir < 0 || dir >= c->nd || side < 0 || side > 1) return fail(MFC_ERR_INVALID, "bad halo side");
  if (!c->halo_buf[2 * dir + side]) return fail(MFC_ERR_INVALID, "that side is not a processor boundary");
  if (count < c->b) return fail(MFC_ERR_INVALID, "need buff_size = (weno_order-1)/2 + 2 ghost widths");
  for (int i = 0; i < c->b; ++i)
    if (!(widths[i] > 0.0)) return fail(MFC_ERR_INVALID, "ghost widths must be positive");
  c->ghost_w[dir][side].assign(widths, widths + c->b);
  // rebuild this context's grid tables with the neighbour's widths
  mfc_params q = c->prm;
  q.x_cb = c->cb_host[0].data();
  q.y_cb = c->nd > 1 ? c->cb_host[1].data() : nullptr;
  q.z_cb = c->nd > 2 ? c->cb_host[2].data() : nullptr;
  const double* gw[3][2];
  for (int d = 0; d < 3; ++d)
    for (int e = 0; e < 2; ++e) gw[d][e] = c->ghost_w[d][e].empty() ? nullptr : c->ghost_w[d][e].data();
  mfc::GridTables gt;
  const std::string why = mfc::build_grid_tables(&q, c->nd, c->n, c->b, gt, gw);
  if (!why.empty()) return fail(MFC_ERR_INVALID, why);
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  MFC_CUDA(cudaMemcpy(c->tables, gt.host.data(), sizeof(double) * gt.host.size(), cudaMemcpyHostToDevice));
  mfc::uniform_records(gt, c->nd, c->n, q.weno_order, q.precision, c->ucoef_found);
  c->ucoef = c->ucoef_enabled ? c->ucoef_found : mfc::UniformCoef{};
  return MFC_OK;
}

int mfc_gpu_halo_pack(mfc_gpu_ctx* c, int stage, int dir, int side, double* dst) {
  if (!c || !dst || dir < 0 || dir >= c->nd || side < 0 || side > 1)
    return fail(MFC_ERR_INVALID, "bad halo pack arguments");
  if (stage < 0 || stage >= c->prm.time_stepper) return fail(MFC_ERR_INVALID, "stage out of range");
  const double* q = stage == 0 ? c->reg[0] : stage == 1 ? c->reg[1] : c->reg[2];
  const int64_t total = strip_elems(c, dir);
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 152 * 8);
  const int wy = c->nd == 2 ? c->n[0] + 2 : c->n[0];
  halo_pack_kernel<<<blocks, 256, 0, c->stream>>>(q, c->S, c->n[0], c->n[1], c->n[2], c->sy, c->sz, c->sv, c->H,
                                                  dir, side, wy, c->halo_buf[0], c->halo_buf[1], c->prm.bc_x_beg,
                                                  c->prm.bc_x_end, c->prm.num_fluids, dst);
  MFC_CUDA(cudaGetLastError());
  c->launches += 1;
  return MFC_OK;
}

int mfc_gpu_set_viscosity(mfc_gpu_ctx* c, const double* re_shear, const double* re_bulk) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  mfc::ViscParams V{};
  const int nf = c->prm.num_fluids;
  for (int f = 0; f < nf; ++f) {
    V.res[0][f] = re_shear ? re_shear[f] : 0.0;
    V.res[1][f] = re_bulk ? re_bulk[f] : 0.0;
    for (int r = 0; r < 2; ++r) V.res_f[r][f] = (float)V.res[r][f];
  }
  for (int r = 0; r < 2; ++r)
    for (int f = 0; f < nf; ++f)
      if (V.res[r][f] > 0.0) V.re_idx[r][V.re_size[r]++] = f;
  const bool on = V.re_size[0] > 0 || V.re_size[1] > 0;
  if (!on) {  // back to the inviscid kernels
    cudaFree(c->visc);
    c->visc = nullptr;
    c->dev.visc = nullptr;
    c->stage = mfc::find_stage(c->nd, nf, c->prm.weno_order, c->prm.precision);
    return MFC_OK;
  }
  if (c->nd > 2) return fail(MFC_ERR_INVALID, "viscous terms are built for 1-D and 2-D cases");
  if (c->chr) return fail(MFC_ERR_INVALID, "the characteristic-field reconstruction is inviscid");
  const mfc::StageEntry* e = mfc::find_stage(c->nd, nf, c->prm.weno_order, c->prm.precision, true);
  if (!e) return fail(MFC_ERR_INVALID, "no viscous kernel compiled for this fluid count / WENO order / precision");
  for (int d = 0; d < c->nd; ++d) V.dcc[d] = c->tables + c->off_dcc[d];
  if (c->wrf) {
    V.fg[0] = c->vg.fg[0];
    V.fg[1] = c->vg.fg[1];
  }
  if (!c->visc && ctx_malloc(c, &c->visc, sizeof(mfc::ViscParams)) != cudaSuccess)
    return fail(MFC_ERR_NOMEM, "viscous parameters");
  MFC_CUDA(cudaMemcpy(c->visc, &V, sizeof(V), cudaMemcpyHostToDevice));
  if (e->prepare() != cudaSuccess) return fail(MFC_ERR_CUDA, "viscous kernel does not fit on this device");
  c->visc_host = V;
  c->dev.visc = c->visc;
  c->stage = e;
  return MFC_OK;
}

namespace {
void free_visc_gradients(mfc_gpu_ctx* c) {
  cudaFree(c->vg.vel);
  cudaFree(c->vg.g);
  for (int k = 0; k < 2; ++k) {
    cudaFree(c->vg.fg[k]);
    cudaFree(c->vg.w[k]);
    cudaFree(c->vg.cf[k]);
  }
  c->vg = mfc::ViscGradBuffers{};
  c->wrf = false;
}
}  // namespace

int mfc_gpu_set_viscous_gradients(mfc_gpu_ctx* c, int weno_re_flux) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (!weno_re_flux) {
    if (c->wrf) {
      MFC_CUDA(cudaStreamSynchronize(c->stream));
      free_visc_gradients(c);
      if (c->visc) {
        c->visc_host.fg[0] = c->visc_host.fg[1] = nullptr;
        MFC_CUDA(cudaMemcpy(c->visc, &c->visc_host, sizeof(c->visc_host), cudaMemcpyHostToDevice));
      }
    }
    return MFC_OK;
  }
  if (!c->visc) return fail(MFC_ERR_INVALID, "weno_Re_flux needs a viscous context (mfc_gpu_set_viscosity first)");
  if (c->prm.precision == MFC_PREC_FP64_FMA)
    return fail(MFC_ERR_INVALID, "weno_Re_flux is built for the FP64, split and gated precisions");
  if (c->prm.weno_order != 5) return fail(MFC_ERR_INVALID, "weno_Re_flux is built for WENO5");
  if (c->has_proc) return fail(MFC_ERR_INVALID, "weno_Re_flux is built without processor boundaries");
  if (c->wrf) return MFC_OK;
  const int nd = c->nd, nx = c->n[0], ny = nd > 1 ? c->n[1] : 1, k = nd * nd;
  // the WENO coefficients and cell widths of the ghost cells up to the
  // reference's viscous buff_size (2*weno_polyn + 2 = 6): cells -3 and n+2
  // enter the gradient reconstructions
  const int bv = 6;
  mfc_params q = c->prm;
  q.x_cb = c->cb_host[0].data();
  q.y_cb = nd > 1 ? c->cb_host[1].data() : nullptr;
  q.z_cb = nullptr;
  mfc::GridTables gt;
  const std::string why = mfc::build_grid_tables(&q, nd, c->n, bv, gt);
  if (!why.empty()) return fail(MFC_ERR_INVALID, why);
  const int bcb[2] = {q.bc_x_beg, q.bc_y_beg}, bce[2] = {q.bc_x_end, q.bc_y_end};
  std::vector<double> w[2];
  for (int d = 0; d < nd; ++d) {
    mfc::AxisHost a;
    a.s = c->n[d] - 1;
    a.b = bv;
    a.cb.assign((size_t)(a.s + 2 * a.b + 2), 0.0);
    a.d.assign((size_t)(a.s + 2 * a.b + 1), 0.0);
    for (int i = -1; i <= a.s; ++i) a.CB(i) = c->cb_host[d][(size_t)(i + 1)];
    mfc::grid_ghosts(a, bcb[d], bce[d]);
    for (int cell = -mfc::kCoefPad; cell <= a.s + mfc::kCoefPad; ++cell) w[d].push_back(a.D(cell));
  }
  cudaError_t e = cudaSuccess;
  auto alloc = [&](double** ptr, size_t count) {
    if (e == cudaSuccess) e = ctx_malloc(c, ptr, sizeof(double) * count);
  };
  const bool fp32 = c->prm.precision == MFC_PREC_SPLIT || c->prm.precision == MFC_PREC_GATED;
  // 2-D split and gated: pairs of the two components, no cell gradients
  const int in8 = fp32 && nd == 2 ? 2 : 1;  // values in 8 bytes
  alloc(&c->vg.vel, (size_t)nd / in8 * (nd > 1 ? ny + 10 : 1) * (nx + 10));
  if (in8 == 1) alloc(&c->vg.g, (size_t)k * (nd > 1 ? ny + 6 : 1) * (nx + 6));
  alloc(&c->vg.fg[0], (size_t)k / in8 * ny * (nx + 1));
  alloc(&c->vg.w[0], w[0].size());
  if (nd > 1) {
    alloc(&c->vg.fg[1], (size_t)k / in8 * (ny + 1) * nx);
    alloc(&c->vg.w[1], w[1].size());
  }
  // split and gated: the reconstructions' FP32 table of each direction
  std::vector<float> cf[2];
  for (int d = 0; fp32 && d < nd; ++d) {
    const size_t stride = w[d].size();  // cells -kCoefPad .. n-1+kCoefPad
    cf[d].resize((mfc::kNumCoef + 1) * stride);
    for (int kk = 0; kk < mfc::kNumCoef; ++kk)
      for (size_t j = 0; j < stride; ++j)
        cf[d][kk * stride + j] = (float)gt.host[gt.off_coef[d] + (size_t)kk * gt.cstride[d] + j];
    for (size_t j = 0; j < stride; ++j) cf[d][mfc::kNumCoef * stride + j] = (float)(1.0 / w[d][j]);
    if (e == cudaSuccess) e = ctx_malloc(c, &c->vg.cf[d], sizeof(float) * cf[d].size());
  }
  if (e != cudaSuccess) {
    free_visc_gradients(c);
    return fail(MFC_ERR_NOMEM, "weno_Re_flux buffers");
  }
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  MFC_CUDA(cudaMemcpy(c->tables, gt.host.data(), sizeof(double) * gt.host.size(), cudaMemcpyHostToDevice));
  for (int d = 0; d < nd; ++d) {
    MFC_CUDA(cudaMemcpy(c->vg.w[d], w[d].data(), sizeof(double) * w[d].size(), cudaMemcpyHostToDevice));
    if (fp32) MFC_CUDA(cudaMemcpy(c->vg.cf[d], cf[d].data(), sizeof(float) * cf[d].size(), cudaMemcpyHostToDevice));
  }
  if (fp32 && nd == 2) {
    c->vg.uniform.on = 1;
    for (int d = 0; d < 2; ++d) {
      const size_t stride = w[d].size();
      for (int kk = 0; kk <= mfc::kNumCoef; ++kk) {
        const float* row = cf[d].data() + (size_t)kk * stride;
        uint32_t b0;
        std::memcpy(&b0, row, 4);
        for (size_t j = 1; j < stride; ++j)
          if (std::memcmp(row + j, row, 4) != 0) c->vg.uniform.on = 0;
        c->vg.uniform.rec[d][kk] = (unsigned long long)b0 << 32 | b0;
      }
    }
  }
  c->visc_host.fg[0] = c->vg.fg[0];
  c->visc_host.fg[1] = c->vg.fg[1];
  MFC_CUDA(cudaMemcpy(c->visc, &c->visc_host, sizeof(c->visc_host), cudaMemcpyHostToDevice));
  c->wrf = true;
  return MFC_OK;
}

int mfc_gpu_set_reconstruction(mfc_gpu_ctx* c, int variables) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (variables != MFC_RECON_PRIMITIVE && variables != MFC_RECON_CHARACTERISTIC)
    return fail(MFC_ERR_INVALID, "variables must be MFC_RECON_PRIMITIVE or MFC_RECON_CHARACTERISTIC");
  const bool chr = variables == MFC_RECON_CHARACTERISTIC && c->prm.weno_order > 1;
  if (chr && c->visc) return fail(MFC_ERR_INVALID, "the characteristic-field reconstruction is inviscid");
  if (chr && c->has_proc)
    return fail(MFC_ERR_INVALID, "the characteristic-field reconstruction is built without processor boundaries");
  const mfc::StageEntry* e =
      mfc::find_stage(c->nd, c->prm.num_fluids, c->prm.weno_order, c->prm.precision, c->visc != nullptr, chr);
  if (!e)
    return fail(MFC_ERR_INVALID, "no characteristic-field kernel compiled for this configuration (FP64, WENO3 "
                                 "or WENO5)");
  MFC_CUDA(e->prepare());
  c->chr = chr;
  c->stage = e;
  return MFC_OK;
}

int mfc_gpu_set_uniform_coefficients(mfc_gpu_ctx* c, int enable, int* in_use) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  c->ucoef_enabled = enable != 0;
  c->ucoef = c->ucoef_enabled ? c->ucoef_found : mfc::UniformCoef{};
  if (in_use) *in_use = c->ucoef.on[0] | (c->ucoef.on[1] << 1) | (c->ucoef.on[2] << 2);
  return MFC_OK;
}

int mfc_gpu_set_monitor(mfc_gpu_ctx* c, int on) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  c->monitor_on = on != 0;
  MFC_CUDA(cudaMemsetAsync(c->monitor, 0, sizeof(unsigned long long), c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

int mfc_gpu_icfl(mfc_gpu_ctx* c, double* icfl_max, int reset) {
  if (!c || !icfl_max) return fail(MFC_ERR_INVALID, "NULL argument");
  unsigned long long bits = 0;
  MFC_CUDA(cudaMemcpyAsync(&bits, c->monitor, sizeof(bits), cudaMemcpyDeviceToHost, c->stream));
  if (reset) MFC_CUDA(cudaMemsetAsync(c->monitor, 0, sizeof(unsigned long long), c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  std::memcpy(icfl_max, &bits, sizeof(double));
  return MFC_OK;
}

int mfc_gpu_run_cfl(mfc_gpu_ctx* c, int num_steps, double cfl, double* dt_inout, double* time_inout) {
  if (!c || !dt_inout || !time_inout) return fail(MFC_ERR_INVALID, "NULL argument");
  if (num_steps < 1 || !(cfl > 0.0) || !(*dt_inout > 0.0)) return fail(MFC_ERR_INVALID, "bad CFL run arguments");
  const bool was_on = c->monitor_on;
  c->monitor_on = true;
  double dt = *dt_inout, t = *time_inout;
  int rc = MFC_OK;
  for (int s = 0; s < num_steps && !rc; ++s) {
    double icfl = 0.0;
    if ((rc = mfc_gpu_icfl(c, &icfl, 1))) break;
    if ((rc = mfc_gpu_tvd_rk(c, dt, 0))) break;
    t += dt;
    if ((rc = mfc_gpu_icfl(c, &icfl, 0))) break;
    if (!(icfl == icfl) || !(icfl > 0.0)) {
      rc = fail(MFC_ERR_STATE, "ICFL is NaN. Exiting ...");
      break;
    }
    dt = dt * (cfl / icfl);  // ICFL of the new state scales with dt
  }
  c->monitor_on = was_on;
  *dt_inout = dt;
  *time_inout = t;
  return rc;
}

int mfc_gpu_run(mfc_gpu_ctx* c, int t_step_start, int t_step_stop, double* dt_inout) {
  if (!c || !dt_inout) return fail(MFC_ERR_INVALID, "NULL argument");
  if (t_step_start < 0 || t_step_stop <= t_step_start)
    return fail(MFC_ERR_INVALID, "Unsupported combination of values of t_step_start and t_step_stop");
  double dt = *dt_inout;
  int t_step = t_step_start;
  double mytime = t_step == 0 ? 0.0 : t_step * dt;
  const double finaltime = t_step_stop * dt;
  for (;;) {
    mytime = mytime + dt;
    int rc = mfc_gpu_tvd_rk(c, dt, t_step == t_step_stop);
    if (rc) return rc;
    if (t_step == t_step_stop) break;
    if ((mytime + dt) >= finaltime) dt = finaltime - mytime;
    t_step = t_step + 1;
  }
  *dt_inout = dt;
  uint32_t flags = 0;
  int rc = mfc_gpu_status(c, &flags, 0);
  if (rc) return rc;
  if (flags & MFC_FLAG_NAN) return fail(MFC_ERR_STATE, "NaN or Inf in the conservative state");
  if (flags & MFC_FLAG_TIMEOUT) return fail(MFC_ERR_STATE, "a TMA staging wait timed out; the state is incomplete");
  if (c->monitor_on) {  // m_data_output.fpp:296-306
    double icfl = 0.0;
    if ((rc = mfc_gpu_icfl(c, &icfl, 0))) return rc;
    if (icfl != icfl) return fail(MFC_ERR_STATE, "ICFL is NaN. Exiting ...");
    if (icfl > 1.0) return fail(MFC_ERR_STATE, "ICFL is greater than 1.0. Exiting ...");
  }
  return MFC_OK;
}

int mfc_gpu_tune(mfc_gpu_ctx* c, int reps, int* variant_out, double* ms_out) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  if (reps < 1) reps = 5;
  uint32_t saved = 0;  // the timing launches must not leave flags behind
  MFC_CUDA(cudaMemcpyAsync(&saved, c->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
  if (c->wrf && c->visc)  // weno_Re_flux: the face gradients that the timed launches read
    MFC_CUDA(mfc::visc_gradients_launch(c->nd, c->prm.num_fluids, c->prm.precision != MFC_PREC_FP64, c->dev, c->vg,
                                        c->reg[0], c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  c->prim_of = nullptr;  // the timed launches use the pairs' buffers
  const mfc::StageEntry* best = nullptr;
  int idx = -1, best_idx = -1;
  float best_ms = 0.f;
  struct Timed {
    const mfc::StageEntry* e;
    int idx;
    float ms;
  };
  std::vector<Timed> timed;
  cudaEvent_t a, b;
  MFC_CUDA(cudaEventCreate(&a));
  MFC_CUDA(cudaEventCreate(&b));
  for (const auto& e : g_reg) {
    if (e.nd != c->nd || e.nf != c->prm.num_fluids || e.wo != c->prm.weno_order || e.prec != c->prm.precision ||
        e.visc != (c->visc != nullptr) || e.chr != c->chr)
      continue;
    ++idx;
    if (e.prepare() != cudaSuccess) continue;
    // first-stage launches read register 0 and write register 1 only; with
    // primitive pairs (of the same state, dt being 0) after the first
    const int64_t pitch = mfc::prim_pitch(c->n[0]);
    mfc::PrimPairs B{nullptr, c->prim[0], pitch, pitch * c->n[1], c->prim[1]};
    auto once = [&] {
      if (c->prim[0] != nullptr && e.launch_prims != nullptr)
        return e.launch_prims(c->dev, c->ucoef, c->reg[0], c->reg[0], c->reg[1], 0.0, mfc::kRkEuler, B, c->stream);
      return e.launch(c->dev, c->ucoef, c->reg[0], c->reg[0], c->reg[1], 0.0, mfc::kRkEuler, c->stream);
    };
    if (once() != cudaSuccess) continue;
    B.in = B.cur = c->prim[0];
    B.out = c->prim[1];
    cudaEventRecord(a, c->stream);
    for (int r = 0; r < reps; ++r) once();
    cudaEventRecord(b, c->stream);
    if (cudaEventSynchronize(b) != cudaSuccess) break;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    ms /= reps;
    if (!best || ms < best_ms) {
      best = &e;
      best_ms = ms;
      best_idx = idx;
    }
    timed.push_back({&e, idx, ms});
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  // a variant that stages its tiles by TMA wins a tie (within 1 %): the copy
  // engine takes the tile loads off the warps at no cost in time
  if (best && !best->tma)
    for (const auto& t : timed)
      if (t.e->tma && t.ms <= best_ms * 1.01f && (!best->tma || t.ms < best_ms)) {
        best = t.e;
        best_ms = t.ms;
        best_idx = t.idx;
      }
  MFC_CUDA(cudaMemcpyAsync(c->status, &saved, sizeof(uint32_t), cudaMemcpyHostToDevice, c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  if (!best) return fail(MFC_ERR_CUDA, "no tile variant could be timed");
  c->stage = best;
  if (variant_out) *variant_out = best_idx;
  if (ms_out) *ms_out = best_ms;
  return MFC_OK;
}

int mfc_gpu_select_variant(mfc_gpu_ctx* c, int variant, int* tx, int* ty, int* threads) {
  if (!c) return fail(MFC_ERR_INVALID, "NULL context");
  int idx = -1;
  for (const auto& e : g_reg) {
    if (e.nd != c->nd || e.nf != c->prm.num_fluids || e.wo != c->prm.weno_order || e.prec != c->prm.precision ||
        e.visc != (c->visc != nullptr) || e.chr != c->chr)
      continue;
    if (++idx != variant) continue;
    if (e.prepare() != cudaSuccess) return fail(MFC_ERR_CUDA, "tile variant does not fit on this device");
    c->stage = &e;
    int ex = e.tx, ey = e.ty, et = e.nt;
    if (e.tile) e.tile(c->n, &ex, &ey, &et);
    if (tx) *tx = ex;
    if (ty) *ty = ey;
    if (threads) *threads = et;
    return MFC_OK;
  }
  return fail(MFC_ERR_INVALID, "no such tile variant for this configuration");
}

int mfc_gpu_variant_features(mfc_gpu_ctx* c, int variant, uint32_t* features) {
  if (!c || !features) return fail(MFC_ERR_INVALID, "NULL argument");
  int idx = -1;
  for (const auto& e : g_reg) {
    if (e.nd != c->nd || e.nf != c->prm.num_fluids || e.wo != c->prm.weno_order || e.prec != c->prm.precision ||
        e.visc != (c->visc != nullptr) || e.chr != c->chr)
      continue;
    if (++idx != variant) continue;
    *features = e.tma ? MFC_VARIANT_TMA : 0u;
    return MFC_OK;
  }
  return fail(MFC_ERR_INVALID, "no such tile variant for this configuration");
}

int mfc_gpu_status(mfc_gpu_ctx* c, uint32_t* flags, int clear) {
  if (!c || !flags) return fail(MFC_ERR_INVALID, "NULL argument");
  MFC_CUDA(cudaMemcpyAsync(flags, c->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
  if (clear) MFC_CUDA(cudaMemsetAsync(c->status, 0, sizeof(uint32_t), c->stream));
  MFC_CUDA(cudaStreamSynchronize(c->stream));
  return MFC_OK;
}

void* mfc_gpu_stream(mfc_gpu_ctx* c) { return c ? (void*)c->stream : nullptr; }

int64_t mfc_gpu_launch_count(const mfc_gpu_ctx* c) { return c ? c->launches : 0; }

int mfc_gpu_snapshot(mfc_gpu_ctx* c, int slot) {
  if (!c || slot < 0 || slot > 1) return fail(MFC_ERR_INVALID, "bad snapshot slot");
  const int64_t cells = (int64_t)c->n[0] * c->n[1] * c->n[2];
  const size_t bytes = (size_t)c->S * cells * sizeof(double);
  if (!c->copy_stream) {
    MFC_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
    MFC_CUDA(cudaEventCreateWithFlags(&c->snap_staged, cudaEventDisableTiming));
  }
  if (!c->snap_host[slot]) {
    if (ctx_malloc(c, &c->snap_dev[slot], bytes) != cudaSuccess) return fail(MFC_ERR_NOMEM, "snapshot staging buffer");
    if (cudaMallocHost(&c->snap_host[slot], bytes) != cudaSuccess) return fail(MFC_ERR_NOMEM, "pinned snapshot slot");
    MFC_CUDA(cudaEventCreateWithFlags(&c->snap_done[slot], cudaEventDisableTiming));
  }
  // the slot's staging buffer is reused: its previous copy-out must have left it
  if (c->snap_pending[slot]) MFC_CUDA(cudaStreamWaitEvent(c->stream, c->snap_done[slot], 0));
  // register 0 -> contiguous staging copy, in stream order with the time steps
  const bool planes_contiguous = c->sz == c->sy * c->n[1];
  for (int v = 0; v < c->S; ++v) {
    double* dst = c->snap_dev[slot] + v * cells;
    if (planes_contiguous) {
      MFC_CUDA(cudaMemcpy2DAsync(dst, (size_t)c->n[0] * 8, c->reg[0] + v * c->sv, (size_t)c->sy * 8,
                                 (size_t)c->n[0] * 8, (size_t)c->n[1] * c->n[2], cudaMemcpyDeviceToDevice,
                                 c->stream));
    } else {
      for (int z = 0; z < c->n[2]; ++z)
        MFC_CUDA(cudaMemcpy2DAsync(dst + (int64_t)z * c->n[0] * c->n[1], (size_t)c->n[0] * 8,
                                   c->reg[0] + v * c->sv + z * c->sz, (size_t)c->sy * 8, (size_t)c->n[0] * 8,
                                   (size_t)c->n[1], cudaMemcpyDeviceToDevice, c->stream));
    }
  }
  MFC_CUDA(cudaEventRecord(c->snap_staged, c->stream));
  // staging -> pinned host on the copy stream; later steps on c->stream overlap with it
  MFC_CUDA(cudaStreamWaitEvent(c->copy_stream, c->snap_staged, 0));
  MFC_CUDA(cudaMemcpyAsync(c->snap_host[slot], c->snap_dev[slot], bytes, cudaMemcpyDeviceToHost, c->copy_stream));
  MFC_CUDA(cudaEventRecord(c->snap_done[slot], c->copy_stream));
  c->snap_pending[slot] = true;
  return MFC_OK;
}

int mfc_gpu_snapshot_wait(mfc_gpu_ctx* c, int slot, const double** host_q) {
  if (!c || slot < 0 || slot > 1 || !host_q) return fail(MFC_ERR_INVALID, "bad snapshot slot");
  if (!c->snap_host[slot]) return fail(MFC_ERR_INVALID, "no snapshot was taken into this slot");
  if (c->snap_pending[slot]) {
    MFC_CUDA(cudaEventSynchronize(c->snap_done[slot]));
    c->snap_pending[slot] = false;
  }
  *host_q = c->snap_host[slot];
  return MFC_OK;
}

int mfc_gpu_finalize(mfc_gpu_ctx* c) {
  if (!c) return MFC_OK;
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->copy_stream) {
    cudaStreamSynchronize(c->copy_stream);
    cudaStreamDestroy(c->copy_stream);
  }
  if (c->snap_staged) cudaEventDestroy(c->snap_staged);
  for (int k = 0; k < 6; ++k) cudaFree(c->halo_buf[k]);
  cudaFree(c->halo_table);
  cudaFree(c->visc);
  for (int s2 = 0; s2 < 2; ++s2) {
    if (c->snap_done[s2]) cudaEventDestroy(c->snap_done[s2]);
    if (c->snap_host[s2]) cudaFreeHost(c->snap_host[s2]);
    cudaFree(c->snap_dev[s2]);
  }
  cudaFree(c->state);
  cudaFree(c->rhs);
  cudaFree(c->tables);
  cudaFree(c->status);
  cudaFree(c->work);
  if (c->nd < 3) cudaFree(c->prim[0]);  // 3-D: part of work
  cudaFree(c->scratch);
  cudaFree(c->vg.vel);
  cudaFree(c->vg.g);
  for (int k = 0; k < 2; ++k) {
    cudaFree(c->vg.fg[k]);
    cudaFree(c->vg.w[k]);
    cudaFree(c->vg.cf[k]);
  }
  cudaFree(c->gate_w);
  cudaFree(c->gate_flags);
  cudaFree(c->monitor);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return MFC_OK;
}

}  // extern "C"

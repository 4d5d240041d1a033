// Kernels of the grouped AM step (many independent problems per launch).
//
// Included by am24_kernels.cu after its anonymous namespace: every kernel
// here runs the same per-column bodies as the one-problem step (gathers,
// densify, split-K reduction, selects, finalize), on the work items of one
// list of the step's plan, with a grid sized to the GPU (a block walks items
// blockIdx.x, blockIdx.x + gridDim.x, ...).  The plan kernel writes the lists
// at the start of each step from every live problem's control words, so the
// lists only hold problems that still iterate, and each problem lands in the
// lists of the path its previous step chose (sparse gather, dense product,
// which select, which operand scheme).

// ------------------------------------------------------------ plan
constexpr int PLAN_THREADS = 1024;

__device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Work items of problem P in list l this step (0: not a member).  Also used
// by the host-side capacity checks through the same rules.
__device__ int plan_items(const GProblem &P, int l) {
  const uint32_t gate = P.ctl[GCTL_GATE];
  const bool dense = gate > P.sparse_cap;
  const bool wide = P.m > GATHER_NARROW;
  const int pairs1 = (P.m_tiles1 + 1) >> 1, pairs2 = (P.m_tiles2 + 1) >> 1;
  switch (l) {
    case GL_GATHER: return !dense && !wide ? P.k : 0;
    case GL_LIST: case GL_FINISH: return !dense && wide ? P.k : 0;
    case GL_TILE: return !dense && wide ? gather_tiles(P.ldm) * gather_groups(P.k) : 0;
    case GL_DENSE: return dense ? P.k : 0;
    case GL_SEL_HARD: return P.formulation <= 1 ? P.k : 0;
    case GL_SEL_SCAN: return (P.formulation == 2 || P.formulation == 3) && !P.l1_exact ? P.k : 0;
    case GL_SEL_EXACT: return (P.formulation == 2 || P.formulation == 3) && P.l1_exact ? P.k : 0;
    case GL_SUPPORT: return P.mixed ? P.k : 0;
    case GL_FIN: return ceil_div(P.k, FIN_STARTS);
    case GL_GEMM1_64: case GL_GEMM1_128: case GL_GEMM1_256:
      return (dense && P.bn == (64 << (l - GL_GEMM1_64))) ? P.splits1 * pairs1 * P.n_tiles1 : 0;
    case GL_RAW_64: case GL_RAW_128: case GL_RAW_256:
      return (P.formulation <= 3 && P.bn == (64 << (l - GL_RAW_64))) ? pairs2 * P.n_tiles2 : 0;
    case GL_PL1_64: case GL_PL1_128: case GL_PL1_256:
      return (P.formulation >= 6 && P.bn == (64 << (l - GL_PL1_64))) ? pairs2 * P.n_tiles2 : 0;
    case GL_PL0_64: case GL_PL0_128: case GL_PL0_256:
      return ((P.formulation == 4 || P.formulation == 5) && P.bn == (64 << (l - GL_PL0_64)))
                 ? pairs2 * P.n_tiles2 : 0;
  }
  return 0;
}

// One block.  For every live problem that has not stopped: its step set-up (this
// step's gate from the last step's count, the batch maximum cleared, the operand
// scheme of V = B^T Z from its MIXED phase) and its place in the list of active
// problems, in slot order; then one warp per work list walks that list: the
// members, compacted in the same order, with exclusive item prefixes.  Counts
// the step and the problems that run it.  A chain of dependent loads and scans:
// 1024 slots, 16 active in 6 us (39 when the whole block scanned the slots list
// by list).
__global__ void __launch_bounds__(PLAN_THREADS) group_plan_kernel(GroupDev g) {
  __shared__ int wsum[PLAN_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int active = 0;
  for (int base = 0; base < g.cap; base += PLAN_THREADS) {
    const int p = base + tid < g.cap ? g.order[base + tid] : g.cap;
    bool act = false;
    if (p < g.cap) {
      GProblem &P = g.probs[p];
      if (P.live && P.ctl[CTL_STOP] == 0u) {
        act = true;
        P.ctl[GCTL_GATE] = P.ctl[GCTL_NEXT];
        P.ctl[GCTL_NEXT] = 0u;
        *P.max_err = 0.f;
        const bool low = P.mixed && P.phase[0] == 0u;
        P.ctl[GCTL_SCHEME] = low ? GS_FP16X1 : (P.mode == 1 ? GS_FP16X2A : GS_FP16X3);
      }
    }
    const uint32_t bits = __ballot_sync(FULL, act);
    __syncthreads();  // wsum of the previous round has been read
    if (lane == 0) wsum[w] = __popc(bits);
    __syncthreads();
    int at = active + __popc(bits & ((1u << lane) - 1u));
    for (int i = 0; i < PLAN_THREADS / 32; i++) {
      if (i < w) at += wsum[i];
      active += wsum[i];
    }
    if (act) g.active[at] = p;
  }
  __syncthreads();  // the block's own writes (active, gates) are read below
  static_assert(GL_COUNT <= PLAN_THREADS / 32, "a warp per list");
  if (w < GL_COUNT) {
    int members = 0, total = 0;
    for (int base = 0; base < active; base += 32) {
      const int p = base + lane < active ? g.active[base + lane] : -1;
      const int items = p >= 0 ? plan_items(g.probs[p], w) : 0;
      int it = items;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int b = __shfl_up_sync(FULL, it, o);
        if (lane >= o) it += b;
      }
      const uint32_t in = __ballot_sync(FULL, items > 0);
      if (items > 0) {
        const int pos = members + __popc(in & ((1u << lane) - 1u));
        g.prob[(size_t)w * g.cap + pos] = p;
        g.pref[(size_t)w * (g.cap + 1) + pos] = total + it - items;
      }
      members += __popc(in);
      total += __shfl_sync(FULL, it, 31);
    }
    if (lane == 0) {
      g.plan->n[w] = members;
      g.plan->total[w] = total;
      g.pref[(size_t)w * (g.cap + 1) + members] = total;
    }
  }
  if (tid < GL_COUNT + 1) g.plan->next[tid] = 0;
  if (tid == 0) {
    g.plan->active = active;
    g.plan->loops += 1;
  }
}

// ------------------------------------------------------------ per-column kernels
// The item loop of one list: fn(problem, local item) for every item of list l.
// Blocks take items from the list's counter, so the widest problems' items
// (listed first) start first and no block idles while another holds a queue.
template <class Fn>
__device__ __forceinline__ void for_items(const GroupDev &g, int l, Fn fn, int counter = -1) {
  __shared__ int taken;
  const int total = g.plan->total[l];
  const int np = g.plan->n[l];
  const int *pref = g.pref + (size_t)l * (g.cap + 1);
  const int *prob = g.prob + (size_t)l * g.cap;
  for (;;) {
    if (threadIdx.x == 0) taken = atomicAdd(&g.plan->next[counter < 0 ? l : counter], 1);
    __syncthreads();
    const int it = taken;
    __syncthreads();
    if (it >= total) break;
    const int i = find_item(pref, np, it);
    const int p = __ldg(prob + i);
    const int local = it - __ldg(pref + i);
    // self-check: the plan only lists live problems' items
    if (np <= 0 || p < 0 || p >= g.cap || !g.probs[p].live || local < 0 ||
        local >= __ldg(pref + i + 1) - __ldg(pref + i)) {
      if (threadIdx.x == 0) atomicCAS(&g.plan->status, 0, (int)DEV_ERR_GROUP_ITEM);
      continue;  // uniform over the block
    }
    fn(g.probs[p], local);
    __syncthreads();  // shared memory is reused by the next item
  }
}

__device__ __forceinline__ ZOut z_out(const GProblem &P, int j) {
  return z_out(j, P.ldm, P.Z_hi, nullptr, P.Z_b, P.Z_h, P.zplane, P.z_scale, P.fz);
}

__global__ void __launch_bounds__(GATHER_THREADS) g_gather_narrow_kernel(GroupDev g) {
  for_items(g, GL_GATHER, [](const GProblem &P, int j) {
    gather_narrow_body(P.mode, P.Bc, P.ldm, P.m, P.ldn, P.Vx, P.vmask, z_out(P, j), j);
  });
}

// the lists take the dense planes' place (not read on sparse steps)
__global__ void __launch_bounds__(GATHER_THREADS) g_gather_list_kernel(GroupDev g) {
  for_items(g, GL_LIST, [](const GProblem &P, int j) {
    gather_list_body(P.ldn, P.Vx, P.vmask, P.sparse_cap, reinterpret_cast<int2 *>(P.V_h), j);
  });
}

__global__ void __launch_bounds__(GATHER_THREADS) g_gather_tile_kernel(GroupDev g) {
  for_items(g, GL_TILE, [](const GProblem &P, int item) {
    gather_tile_body(P.Bc, P.ldm, P.ldn, P.k, reinterpret_cast<const int2 *>(P.V_h), P.Z_hi, item);
  });
}

// dense steps before Z = B V: the FP16 planes of V
__global__ void __launch_bounds__(DENSIFY_THREADS, DENSIFY_BLOCKS_PER_SM)
    g_densify_kernel(GroupDev g) {
  for_items(g, GL_DENSE, [](const GProblem &P, int j) {
    densify_fp16_body(P.Vx, P.vmask, P.ldn, P.n, P.V_h, (size_t)P.k * P.ldn, P.v_scale,
                      P.ctl + GCTL_GATE, P.sparse_cap, P.ctl + CTL_STOP, j);
  });
}

// after Z = B V: the split-K sum of dense steps, the end of the tiled gathers
__global__ void __launch_bounds__(256) g_z_reduce_kernel(GroupDev g) {
  for_items(g, GL_DENSE, [](const GProblem &P, int j) {
    z_reduce_body(P.mode, P.ws, P.splits1, P.m_tiles1, P.n_tiles1, P.bn, P.m, z_out(P, j), j);
  }, GL_COUNT);
  for_items(g, GL_FINISH,
            [](const GProblem &P, int j) { z_finish_body(P.mode, P.m, z_out(P, j)); });
}

__global__ void __launch_bounds__(HARD_THREADS) g_hard_select_kernel(GroupDev g) {
  for_items(g, GL_SEL_HARD, [](const GProblem &P, int j) {
    hard_select_body(P.Vraw, P.ldn, P.n, P.constraint, P.Vx, P.nnz, P.vmask,
                     P.sel_hint, P.cmask, j);
  });
}

template <bool EXACT>
__global__ void __launch_bounds__(SOFT_THREADS, 4) g_soft_select_kernel(GroupDev g) {
  for_items(g, EXACT ? GL_SEL_EXACT : GL_SEL_SCAN, [](const GProblem &P, int j) {
    soft_select_body<EXACT>(P.Vraw, P.ldn, P.n, P.constraint, P.Vx, P.nnz, P.vmask,
                            P.sel_hint, P.cmask, j);
  });
}

// MIXED: per start, whether its support (non-zero mask) changed this step, by
// a 64-bit hash of the mask words (splitmix64 of (word index, word), summed,
// so that the order of the additions does not matter); then the stability
// count and, by the problem's last item, the phase switch (support_kernel's
// rule).  The hash of a column that changed equals the previous one with
// probability 2^-64.
__global__ void __launch_bounds__(256) g_support_kernel(GroupDev g) {
  __shared__ unsigned long long red[8];
  for_items(g, GL_SUPPORT, [&](const GProblem &P, int j) {
    const int words = P.ldn >> 5;
    const uint32_t *a = P.vmask + (size_t)j * words;
    unsigned long long h = 0ull;
    for (int wd = threadIdx.x; wd < words; wd += blockDim.x)
      h += splitmix64(((uint64_t)(uint32_t)wd << 32) | a[wd]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(FULL, h, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = h;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0ull;
      for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
      const bool same = P.mask_hash[j] == t;
      P.mask_hash[j] = t;
      // no start counts as stable during the FP32 lead-in (phase[0] >= 2)
      const bool lead = *reinterpret_cast<volatile uint32_t *>(P.phase) >= 2u;
      const uint32_t st = (same && !lead) ? min(P.stable[j] + 1u, 0x7FFFFFFFu) : 0u;
      P.stable[j] = st;
      if (st >= P.k_stable) atomicAdd(&P.ctl[GCTL_SUPPORT], 1u);
      __threadfence();
      if (atomicAdd(&P.ctl[GCTL_SBLOCKS], 1u) == (uint32_t)P.k - 1) {
        __threadfence();
        const uint32_t count = atomicExch(&P.ctl[GCTL_SUPPORT], 0u);
        const uint32_t ph = P.phase[0];
        P.phase[3] = ph;
        P.phase[0] = mixed_next_phase(ph, count >= P.need_stable);
        P.ctl[GCTL_SBLOCKS] = 0u;
      }
    }
  });
}

// Per start the objective, change and batch maximum (finalize_start); the
// problem's last item closes its step: counts it, keeps the largest change and
// sets the stop word after the step the reference's batch loop ends on (it > 0
// in the refinement phase with the largest change below the tolerance), after
// its max_iter-th step, or when a device-side wait gave up.
__global__ void __launch_bounds__(256) g_finalize_kernel(GroupDev g) {
  for_items(g, GL_FIN, [&](const GProblem &P, int item) {
    FinalizeArgs a;
    a.k = P.k;
    a.formulation = P.formulation;
    a.parts = P.parts;
    a.it = (int)P.ctl[CTL_STEPS];
    a.store_all = 0;
    a.log_shift = 0;
    a.log_capacity = 0;
    a.tolerance = P.tolerance;
    a.fz = P.fz;
    a.obj_part = P.obj_part;
    a.nnz_part = P.nnz_part;
    a.nnz_sel = P.nnz;
    a.val = P.val;
    a.err = P.err;
    a.max_err = P.max_err;
    a.next_nnz = P.ctl + GCTL_NEXT;
    a.max_nnz = a.planes_nnz = a.host_stop = nullptr;  // the plan hands the count on
    a.iters = nullptr;
    a.cards = nullptr;
    a.ctl = P.ctl;
    a.phase = P.mixed ? P.phase : nullptr;
    a.status = P.status;
    a.stop_check = 1;
    const int j = item * FIN_STARTS + (threadIdx.x >> 5);
    if (j < P.k) finalize_start(a, j, threadIdx.x & 31);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const int items = ceil_div(P.k, FIN_STARTS);
      if (atomicAdd(&P.ctl[CTL_BLOCKS], 1u) == (uint32_t)items - 1) {
        __threadfence();
        const float me = *reinterpret_cast<volatile float *>(P.max_err);
        const bool refined = !P.mixed || P.phase[3] != 0u;
        const uint32_t steps = P.ctl[CTL_STEPS] + 1u;
        P.ctl[CTL_STEPS] = steps;
        if (!refined) P.ctl[CTL_LOW_STEPS] += 1u;
        P.ctl[CTL_MAX_ERR] = __float_as_uint(me);
        if ((a.it > 0 && refined && (double)me < P.tolerance) ||
            steps >= (uint32_t)P.max_iter ||
            *reinterpret_cast<const volatile int *>(P.status) != 0)
          P.ctl[CTL_STOP] = 1u;
        P.ctl[CTL_BLOCKS] = 0u;
      }
    }
  });
}

// The WHILE condition of a captured step loop: another step while some live
// problem has not stopped, the launch's step cap is not reached and no wait
// of a grouped product gave up.  Also writes every slot's state to g.done,
// which a host polls with one copy.
__global__ void __launch_bounds__(256) g_condition_kernel(GroupDev g,
                                                          cudaGraphConditionalHandle handle,
                                                          bool in_graph) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < g.cap; p += blockDim.x) {
    const GProblem &P = g.probs[p];
    uint32_t d = 0u;
    if (P.live) {
      d = *reinterpret_cast<volatile const uint32_t *>(P.ctl + CTL_STOP) == 0u ? 1u : 2u;
      if (d == 1u) any = 1;
    }
    g.done[p] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const GPlan &pl = *g.plan;
    const bool more = any && pl.loops < pl.loop_cap && pl.status == 0;
    if (in_graph) cudaGraphSetConditional(handle, more ? 1u : 0u);
  }
}

// minres_driver.inl -- (P)MINRES launch sequence; included by cudapcg_b200.cu.
// Recurrence of chfem/src/femhmg/cudapcg/solvers/pminres.cu:28-247 (and minres.cu:58-260
// without preconditioner).  Per iteration: the pointwise direction pass finishes alpha, the
// operator pass updates x and r, applies A to z = M^-1 r and finishes delta, beta and the
// stopping test.  r alternates between two buffers (read r, write r'), so chunks are even; the
// Stokes iteration is the three passes of stencil_fluid_mr.cuh, with r in place.

static MrCfg mrcfg() {
  MrCfg cfg;
  const SolveCfg sc = solvecfg();
  cfg.tol = sc.tol; cfg.maxit = sc.maxit; cfg.norm = sc.norm; cfg.precond = sc.precond; cfg.nhmg = sc.nhmg;
  return cfg;
}

// Whether the Stokes records of nr directions are kept per grid node (stencil_fluid_mr.cuh): 8 %
// faster than per fluid node at 96^3 and porosity 0.35, for 32 N nr bytes instead of 32 (nV + nB) nr.
// Not where the grid holds more than four nodes per fluid node (128 bytes per fluid node) or its
// records exceed 16 GiB: what a model that fills the device holds beside its vectors, 48 bytes per
// unknown, is then 32 bytes per fluid node.
static bool fl_by_node(int nr) { return S->N <= 4l * (S->nV + S->nB) && 32l * S->N * nr <= 16l << 30; }
static size_t fl_record_bytes(int nr) { return 32ul * nr * std::max(fl_by_node(nr) ? S->N : S->nV + S->nB, 1l); }

// The Stokes passes (stencil_fluid_mr.cuh) on explicit buffers, nr directions n unknowns apart.  A
// pixel model solves one direction at a time: its blocks do not exist.
static FlMrArgs fl_mr_args(int nr, double* r, double* q, double* s, double* d, double* x, double* z, int fin, bool skip_if_done) {
  return FlMrArgs{r, q, s, d, x, z, S->d_node_of_dof, S->d_bkeys, fl_by_node(nr) ? nullptr : S->d_dof_of_node, S->R, S->C, S->L, S->nV, S->nB, S->nvars,
                  S->cur_sc, RedCtl{}, mrcfg(), fin, skip_if_done};
}
template <int NR>
static bool launch_fl_mr_dir(FlMrArgs a) {
  const int g = pw_grid(S->nvars);
  if (!ensure_reduction(g)) return false;
  a.rc = redctl(g);
  if constexpr (NR == 1)
    if (S->fdim == 2) k_fl_mr_dir<1, 2><<<g, PW_NT, 0, S->stream>>>(a);
  if (S->fdim == 3) k_fl_mr_dir<NR, 3><<<g, PW_NT, 0, S->stream>>>(a);
  S->launches++;
  return cudaPeekAtLastError() == cudaSuccess;
}
template <int NR>
static bool launch_fl_mr_upd(const FlMrArgs& a) {
  const int g = pw_grid(S->nvars);
  if constexpr (NR == 1)
    if (S->fdim == 2) k_fl_mr_upd<1, 2><<<g, PW_NT, 0, S->stream>>>(a);
  if (S->fdim == 3) k_fl_mr_upd<NR, 3><<<g, PW_NT, 0, S->stream>>>(a);
  S->launches++;
  return cudaPeekAtLastError() == cudaSuccess;
}
template <int NR, int DIM, bool GRID>
static void launch_fl_mr_apply_dim(const FlMrArgs& a, int g) {
  if (S->resnorm == CUDAPCG_L2_NORM) k_fl_mr_apply<NR, DIM, false, GRID><<<g, FL_NT, 0, S->stream>>>(a);
  else k_fl_mr_apply<NR, DIM, true, GRID><<<g, FL_NT, 0, S->stream>>>(a);
}
template <int NR>
static bool launch_fl_mr_apply(FlMrArgs a) {
  const int g = pw_grid(S->nV + S->nB);
  if (!ensure_reduction(g)) return false;
  a.rc = redctl(g);
  const bool grid = !a.dof_of_node;
  if constexpr (NR == 1)
    if (S->fdim == 2) grid ? launch_fl_mr_apply_dim<1, 2, true>(a, g) : launch_fl_mr_apply_dim<1, 2, false>(a, g);
  if (S->fdim == 3) grid ? launch_fl_mr_apply_dim<NR, 3, true>(a, g) : launch_fl_mr_apply_dim<NR, 3, false>(a, g);
  S->launches++;
  return cudaPeekAtLastError() == cudaSuccess;
}

// Operator pass of (P)MINRES on explicit buffers: r' = r - alpha q into rout, s = A M^-1 r',
// x += alpha d, with the scalars of S->cur_sc.
template <typename T>
static bool launch_mr_op_buf(const T* rin, T* rout, const T* q, T* s, double* x, const T* d, int fin, bool skip_if_done) {
  const MrCfg cfg = mrcfg();
  if (S->fluid) {
    if constexpr (sizeof(T) == 8) {  // r is updated in place (rout unused)
      if (!launch_fl_mr_upd<1>(fl_mr_args(1, (T*)rin, (T*)q, s, (T*)d, x, S->fl_z, fin, skip_if_done))) return false;
      return launch_fl_mr_apply<1>(fl_mr_args(1, (T*)rin, (T*)q, s, (T*)d, x, S->fl_z, fin, skip_if_done));
    }
    set_err("operator pass", "Stokes models solve in FP64");
    return false;
  } else if (S->dim2) {
    const int nb = d2_ctas();
    if (!ensure_reduction(nb)) return false;
    if (S->nd == 1) {
      TeArgs<1, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat, S->R, S->C, 1, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      sdf_args(a);
      k_2d_apply<1, T, TE_MR><<<nb, dim3(T2_TR, T2_TC), t2_smem_bytes<1, T>(), S->stream>>>(a);
    } else {
      TeArgs<2, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat, S->R, S->C, 1, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      sdf_args(a);
      k_2d_apply<2, T, TE_MR><<<nb, dim3(T2_TR, T2_TC), t2_smem_bytes<2, T>(), S->stream>>>(a);
    }
  } else if (md_applies()) {
    return S->nd == 1 ? launch_md<1, T, TE_MR>(rin, q, rout, s, x, d, fin, skip_if_done, cfg)
                      : launch_md<3, T, TE_MR>(rin, q, rout, s, x, d, fin, skip_if_done, cfg);
  } else if (asm_applies()) {
    int nb;
    cudaError_t e;
    if (S->nd == 1) {
      nb = asm_te_ctas<1, T, TE_MR>(S->R, S->C, S->L, num_sms());
      if (nb < 1 || !ensure_reduction(nb)) return false;
      TeArgs<1, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat, S->R, S->C, S->L, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      e = asm_te_launch<1, T, TE_MR>(a, tabdev<T>(), nb, S->stream);
    } else {
      nb = asm_te_ctas<3, T, TE_MR>(S->R, S->C, S->L, num_sms());
      if (nb < 1 || !ensure_reduction(nb)) return false;
      TeArgs<3, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat, S->R, S->C, S->L, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      e = asm_te_launch<3, T, TE_MR>(a, tabdev<T>(), nb, S->stream);
    }
    S->launches++;
    if (e != cudaSuccess) { set_err("operator pass", cudaGetErrorString(e)); return false; }
    return true;
  } else {
    const dim3 block(TE_TR, TE_TC);
    if (S->nd == 1) {
      const size_t sm = te_smem_bytes<1, T>(S->nmat);
      const int nb = te_ctas(k_te_apply<1, T, TE_MR>, sm);
      if (!ensure_reduction(nb)) return false;
      TeArgs<1, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat,
                     S->R, S->C, S->L, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      sdf_args(a);
      k_te_apply<1, T, TE_MR><<<nb, block, sm, S->stream>>>(a);
    } else {
      const size_t sm = te_smem_bytes<3, T>(S->nmat);
      const int nb = te_ctas(k_te_apply<3, T, TE_MR>, sm);
      if (!ensure_reduction(nb)) return false;
      TeArgs<3, T> a{rin, q, rout, s, x, d, S->d_keys, Kdev<T>(), S->nmat,
                     S->R, S->C, S->L, S->cur_sc, redctl(nb), fin, skip_if_done, cfg};
      sdf_args(a);
      k_te_apply<3, T, TE_MR><<<nb, block, sm, S->stream>>>(a);
    }
  }
  S->launches++;
  return cudaPeekAtLastError() == cudaSuccess;
}
template <typename T>
static bool launch_mr_op(const T* rin, T* rout, int fin, bool skip_if_done) {
  return launch_mr_op_buf<T>(rin, rout, (const T*)S->q, (T*)S->s, S->x, (const T*)S->d0, fin, skip_if_done);
}

template <typename T>
static bool launch_mr_dir(const T* rcur) {
  if (S->fluid) {
    if constexpr (sizeof(T) == 8) return launch_fl_mr_dir<1>(fl_mr_args(1, (T*)rcur, (T*)S->q, (T*)S->s, (T*)S->d0, S->x, S->fl_z, FIN_ALPHA, true));
    set_err("direction pass", "Stokes models solve in FP64");
    return false;
  } else {
    const int g = pw_grid(S->N);
    if (!ensure_reduction(g)) return false;
    if (S->dim2 && S->nd == 2) {  // 2D elastic: the Jacobi diagonal from invd only
      MrDirTe<2, T> a{(T*)S->d0, (T*)S->q, rcur, (const T*)S->s, S->d_keys, Kdev<T>(), 0, S->N, S->cur_sc, redctl(g), S->precond, S->d_invd};
      k_te_mr_dir<2, T><<<g, PW_NT, 0, S->stream>>>(a);
    } else if (S->nd == 1) {
      MrDirTe<1, T> a{(T*)S->d0, (T*)S->q, rcur, (const T*)S->s, S->d_keys, Kdev<T>(), S->dim2 ? 0 : S->nmat, S->N, S->cur_sc, redctl(g), S->precond, S->d_invd};
      k_te_mr_dir<1, T><<<g, PW_NT, 0, S->stream>>>(a);
    } else {
      MrDirTe<3, T> a{(T*)S->d0, (T*)S->q, rcur, (const T*)S->s, S->d_keys, Kdev<T>(), S->nmat, S->N, S->cur_sc, redctl(g), S->precond, S->d_invd};
      k_te_mr_dir<3, T><<<g, PW_NT, 0, S->stream>>>(a);
    }
  }
  S->launches++;
  return cudaPeekAtLastError() == cudaSuccess;
}

template <typename T>
static bool enqueue_minres_iteration(int parity) {
  // thermal / elastic: the residual alternates between two buffers (Stokes updates it in place)
  const T* rcur = (const T*)(parity && !S->fluid ? S->r2 : S->r);
  T* rnext = (T*)(parity ? S->r : S->r2);
  return launch_mr_dir<T>(rcur) && launch_mr_op<T>(rcur, rnext, FIN_MR_STEP, true);
}

template <typename T>
static bool solve_minres_device() {
  if (!ensure_reduction(needed_blocks())) return false;
  CKV(cudaMemsetAsync(S->d_ticket, 0, sizeof(unsigned), S->stream));
  CKV(cudaMemsetAsync(S->cur_sc, 0, sizeof(DevScalars), S->stream));
  const size_t n = (size_t)S->nvars;
  if (!S->x0_set) CKV(cudaMemsetAsync(S->x, 0, n * 8, S->stream));
  CKV(cudaMemsetAsync(S->q, 0, n * sizeof(T), S->stream));
  CKV(cudaMemsetAsync(S->d0, 0, n * sizeof(T), S->stream));
  CKV(cudaEventRecord(S->ev0, S->stream));
  // zero-guess reference (pminres.cu:58-79): res0 = r.M^-1 r, s = A M^-1 r, delta0 = z.s.
  // alpha is 0 here, so r' = r and x is unchanged.
  if (!launch_mr_op<T>((const T*)S->r, (T*)S->r2, FIN_MR_INIT, false)) return false;
  if (S->x0_set) {  // pminres.cu:81-98: r = b - A x0 (FP64 apply), then the same evaluation
    if (!residual_from_x<T>()) return false;
    if (!launch_mr_op<T>((const T*)S->r, (T*)S->r2, FIN_MR_X0, true)) return false;
  }
  CKV(cudaEventRecord(S->ev1, S->stream));
  if (!run_chunks<T>(true)) return false;
  CKV(cudaEventRecord(S->ev2, S->stream));
  CKV(cudaEventSynchronize(S->ev2));
  float ms1 = 0, ms2 = 0;
  cudaEventElapsedTime(&ms1, S->ev0, S->ev1);
  cudaEventElapsedTime(&ms2, S->ev1, S->ev2);
  S->setup_dev_s = ms1 * 1e-3;
  S->solve_dev_s = ms2 * 1e-3;
  return true;
}

/*
 * Constrained transport (in.par Constrained_Transport 1; bfields.c,
 * riemann.c:73-110 and 175-213, onestep.c:140-185) as order-preserving
 * per-cell and per-face kernels.  CT_MODE 1 (2D: the in-plane field) and
 * CT_MODE 2 (3D: also the z faces, the E_phi edges and make_edge_adjust).
 * The edge arithmetic runs in the bulk real type R (FP32 in the mixed form);
 * the face fluxes Phi and their updates E dl dt stay FP64, so CT keeps the
 * discrete div B in both forms.
 *
 * The reference keeps the magnetic flux of every r- or z-face in one slot of
 * the cell that "owns" the face (the face ending at the cell's piph: r faces
 * LRtype 0 -> L->Phi[2], 1 -> R->Phi[1]; z faces L->Phi[4], R->Phi[3];
 * get_phi_pointer, bfields.c:734-758) and the flux through the cell's phi
 * face at piph in Phi[0].  A cell owns exactly one face of each track beside
 * it; the face builder records it (consL / consR, consZL / consZR), so every
 * scatter of bfields.c becomes a gather:
 *
 *   k_update     phi faces' (Ez, Br, Er, Bz) from flux_to_E (also on the
 *                ghost annuli next to the real ones, misc.c:382-397)
 *   k_flux_t     r and z faces' (Erz, Brz, E_phi)
 *   k_ct_edges   each cell's edge values E[0..7], B[0..7]: the phi faces'
 *                half values plus the r and z faces' fractions, in face order
 *   k_ct_faces   avg_Efields (bfields.c:392-644: phi average, then the
 *                face's interpolation) and subtract_advective_B_fluxes
 *                (:646-690) for each face's owner edge, then E dl dt
 *   k_ct_line    make_edge_adjust's 4-way merge (bfields.c:888-1127) as a
 *                merge path: each cell finds its step in the merge of every
 *                edge line it borders (from the face lists of the two tracks
 *                it shares with the line and one binary search for the
 *                diagonal annulus), re-evaluates get_which4 there and writes
 *                that step's E_phi dl dt
 *   k_ct_update  update_B_fluxes (:313-382) and make_edge_adjust on each
 *                cell's slots: a slot gets its own face's term and the
 *                previous face's, in the order the track loop applies them,
 *                then the edge steps of its two lines, in line order; Phi[0]
 *                the owned faces' terms; then move_cells
 *   k_ct_flag    check_flipped (:693-731) on the moved cells
 *   k_ct_flip    flip_fluxes (:760-814): one warp per track, flagged faces
 *                in order by one lane (LRtype toggles carry to later ones)
 *   ct_cons_B    B_faces_to_cells type 1 (:88-309) before calc_prim
 *
 * Values the reference leaves stale (edge fields and E_phi of annuli and
 * faces outside the CT flux ranges) are zero here; they reach only slots of
 * ghost cells' faces that no real cell reads.  The r-pole branches of
 * avg_Efields (NgRa/NgRb = 0) write edges that no face owns, so they are not
 * evaluated; the z-pole branches (NgZa/NgZb = 0 in 3D) reach the z faces the
 * bottom layer's cells own above them and the top layer's own below them:
 * k_ct_faces keeps those faces' E per owner and k_ct_zpole writes their X
 * from the annulus mean.
 */
#pragma once
#include "disco_kernels.cuh"

namespace disco {

/* annuli whose phi faces phi_flux evaluates under CT (misc.c:382-397) */
__device__ __forceinline__ bool ct_phi_annulus(const DiskParams &P, int j, int k){
   int jmin = P.NgRa == 0 ? 0 : P.NgRa-1, jmax = P.NgRb == 0 ? P.Nr : P.Nr-P.NgRb+1;
   int kmin = P.NgZa == 0 ? 0 : P.NgZa-1, kmax = P.NgZb == 0 ? P.Nz : P.Nz-P.NgZb+1;
   return j >= jmin && j < jmax && k >= kmin && k < kmax;
}

/* the slot holding face f's flux under its current LRtype (z: zf) */
template<class R>
__device__ __forceinline__ double *ct_slot(const ViewT<R> &v, double *base, int f, bool zf){
   if( zf ) return v.fLR[f] == 0 ? base + AT_PHI(4, v.fL[f]) : base + AT_PHI(3, v.fR[f]);
   return v.fLR[f] == 0 ? base + AT_PHI(2, v.fL[f]) : base + AT_PHI(1, v.fR[f]);
}

/* fn(f) for each face of cell i's runs in track t, in face order */
template<class R, class F>
__device__ __forceinline__ void ct_over_runs(const ViewT<R> &v, const int *cons, int t, int c0,
                                             int np, int i, int I0, F fn){
   Runs rn = cell_runs(v, cons, t, c0, np, i, I0);
   for( int f=rn.s1 ; f<=rn.e1 ; ++f ) fn(f);
   for( int f=rn.s2 ; f<=rn.e2 ; ++f ) fn(f);
}

template<class R>
__global__ void __launch_bounds__(CB, MB_CT_EDGES) k_ct_edges(ViewT<R> v){
   const CellBlk b = v.cblk[blockIdx.x];
   int a = b.x, i = b.y + threadIdx.x;
   int np = b.np;
   if( i >= np ) return;
   int c0 = b.c0, c = c0 + i;
   int cm = c0 + (i == 0 ? np-1 : i-1);
   const DiskParams &P = v.dp[b.disk];
   int j = b.j, k = b.k;
   const int ne = v.ct == 2 ? 8 : 4;
   R E[8] = {0,0,0,0,0,0,0,0}, B[8] = {0,0,0,0,0,0,0,0};
   if( ct_phi_annulus(P, j, k) ){
      /* riemann_phi: cL->E[0], E[1] (E[4], E[5]) and cR->E[2], E[3] (E[6],
       * E[7]) = .5 Ez (.5 Er), riemann.c:73-110 */
      R eR = R(.5)*v.pE[c], eL = R(.5)*v.pE[cm];
      R bR = R(.5)*v.pB[c], bL = R(.5)*v.pB[cm];
      E[0] = eR; E[1] = eR; E[2] = eL; E[3] = eL;
      B[0] = bR; B[1] = bR; B[2] = bL; B[3] = bL;
      if( v.ct == 2 ){
         R zR = R(.5)*v.pEr[c], zL = R(.5)*v.pEr[cm];
         R wR = R(.5)*v.pBz[c], wL = R(.5)*v.pBz[cm];
         E[4] = zR; E[5] = zR; E[6] = zL; E[7] = zL;
         B[4] = wR; B[5] = wR; B[6] = wL; B[7] = wL;
      }
      R dph = (R)v.dphi[c];
      int I0 = v.I0[a];
      /* riemann_trans (riemann.c:175-205): as R of the inner (lower) track
       * E[0], E[2] (E[4], E[6]) += .5 Erz fracR; as L of the outer (upper)
       * track E[1], E[3] (E[5], E[7]) += .5 Erz fracL */
      auto add = [&](int lo, int hi) {
         return [&, lo, hi](int f) {
            R fr = (R)v.fdp[f] / dph;
            R xe = R(.5)*v.fEt[f]*fr, xb = R(.5)*v.fBt[f]*fr;
            E[lo] += xe; E[hi] += xe; B[lo] += xb; B[hi] += xb;
         };
      };
      if( j >= 1 ){
         int t = P.trr0 + (j-1) + (P.Nr-1)*k;
         if( v.tr_flux[t] ) ct_over_runs(v, v.consR, t, c0, np, i, I0, add(0, 2));
      }
      if( j <= P.Nr-2 ){
         int t = P.trr0 + j + (P.Nr-1)*k;
         if( v.tr_flux[t] ) ct_over_runs(v, v.consL, t, c0, np, i, I0, add(1, 3));
      }
      if( v.ct == 2 && P.Nz > 1 ){
         if( k >= 1 ){
            int t = P.trz0 + j + P.Nr*(k-1);
            if( v.tr_flux[t] ) ct_over_runs(v, v.consZR, t, c0, np, i, I0, add(4, 6));
         }
         if( k <= P.Nz-2 ){
            int t = P.trz0 + j + P.Nr*k;
            if( v.tr_flux[t] ) ct_over_runs(v, v.consZL, t, c0, np, i, I0, add(5, 7));
         }
      }
   }
#pragma unroll
   for( int s=0 ; s<8 ; ++s ) if( s < ne ){ v.ctE[AT_EDGE(s, c)] = E[s]; v.ctB[AT_EDGE(s, c)] = B[s]; }
}

/* next / previous cell of annulus a (cyclic) */
template<class R>
__device__ __forceinline__ int ct_next(const ViewT<R> &v, int a, int c){
   int o = v.ann_off[a], n = v.ann_np[a];
   return c+1 == o+n ? o : c+1;
}
template<class R>
__device__ __forceinline__ int ct_prev(const ViewT<R> &v, int a, int c){
   int o = v.ann_off[a], n = v.ann_np[a];
   return c == o ? o+n-1 : c-1;
}

template<class R>
__global__ void __launch_bounds__(FB, MB_CT_FACES) k_ct_faces(ViewT<R> v){
   const FaceBlk b = v.fblk[blockIdx.x];
   int t = b.x;
   bool zf = b.dim == 2;
   if( zf && v.ct != 2 ) return;
   int f = b.f0 + b.y + threadIdx.x;
   if( f >= b.f1 ) return;
   int A = b.A, Bn = b.B;
   int d = b.disk;
   const DiskParams &P = v.dp[d];
   int err = 0;
   int L = v.fL[f], Rc = v.fR[f];
   int lr = v.fLR[f];
   int o = lr == 0 ? L : Rc, c2 = lr == 0 ? Rc : L;
   int ao = lr == 0 ? A : Bn, a2 = lr == 0 ? Bn : A;
   int on = ct_next(v, ao, o);
   int c2n = ct_next(v, a2, c2), c2p = ct_prev(v, a2, c2);
   const R *E = v.ctE, *B = v.ctB;
   const size_t s0 = zf ? 4 : 0;          /* r faces use edges 0-3, z faces 4-7 */
   /* the phi average of avg_Efields: edge s of cell c becomes
    * .5 (E[s](c) + E[s+2](c+1)) for the right edges s = 0, 1 and
    * .5 (E[s-2](c-1) + E[s](c)) for the left ones (bfields.c:400-442) */
   double p1 = v.piph[o], p2 = v.piph[c2];
   double dp1 = get_dp(p2, p1, P.Pmax, &err);
   double dp2 = v.dphi[c2] - dp1;
   const R w1 = (R)dp1, w2 = (R)dp2;
   /* owner edge s_o (and its left twin s_o+2); c2's edges s_c, s_c+2 */
   size_t so = lr == 0 ? s0+1 : s0, sc = lr == 0 ? s0 : s0+1;
   R Eo = R(.5)*(E[AT_EDGE(so, o)] + E[AT_EDGE(so+2, on)]);
   R Bo = R(.5)*(B[AT_EDGE(so, o)] + B[AT_EDGE(so+2, on)]);
   R ea = R(.5)*(E[AT_EDGE(sc, c2)] + E[AT_EDGE(sc+2, c2n)]), eb = R(.5)*(E[AT_EDGE(sc, c2p)] + E[AT_EDGE(sc+2, c2)]);
   R ba = R(.5)*(B[AT_EDGE(sc, c2)] + B[AT_EDGE(sc+2, c2n)]), bb = R(.5)*(B[AT_EDGE(sc, c2p)] + B[AT_EDGE(sc+2, c2)]);
   R Eav = ( w2*ea + w1*eb )/(w1+w2);
   R Bav = ( w2*ba + w1*bb )/(w1+w2);
   R fE = R(.5)*(Eo + Eav);
   R fB = R(.5)*(Bo + Bav);
   /* subtract_advective_B_fluxes: the owner's edge moves with its wiph; an
    * r face's edge sits at r_jph[j] (E -= h w B), a z face's at the
    * annulus centroid (E += h w B) */
   int j = b.j, k = b.k;
   const double *rj = v.rj + P.rj0 + 1;
   const double *zk = v.zk + P.zk0 + 1;
   double w = v.wiph[o];
   R Ef;
   double dl;
   if( !zf ){
      double h = rj[j];
      Ef = fE - (R)(h*w)*fB;
      dl = zk[k]-zk[k-1];                         /* r-face dl = dz, faces_alt.c:26-27 */
   }else{
      double h = v.tr_r[t];                        /* centroid_r(r_j, r_j-1) */
      Ef = fE + (R)(h*w)*fB;
      dl = rj[j]-rj[j-1];                         /* z-face dl = dr */
   }
   double dt = v.ds[d].dt*v.dtfac;
   /* avg_Efields' z-pole branch (bfields.c:580-617): without z ghosts the
    * bottom layer's E[5] and the top layer's E[4] become their annulus's
    * mean and B 0 -- the owner's value is kept for k_ct_zpole, which writes
    * these faces' X */
   if( zf && v.ctPole && ((lr == 0 && k == 0 && P.NgZa == 0) ||
                          (lr == 1 && k+1 == P.Nz-1 && P.NgZb == 0)) ){
      v.ctPole[o] = (double)fE;
   }else{
      v.fX[f] = (double)Ef*dl*dt;
   }
   raise_err(v, err);
}

/* The z-pole average (bfields.c:580-617) of pole annulus pl[blockIdx.x]
 * (x: annulus, y: 0 the bottom layer, its cells' upper faces; 1 the top
 * layer, their lower faces): E = the sum of the cells' owned-face E in cell
 * order over Np, B = 0, so the advective term vanishes and each owned face
 * takes X = E dl dt. */
template<class R>
__global__ void __launch_bounds__(CB) k_ct_zpole(ViewT<R> v, const int2 *pl){
   __shared__ double s_E;
   const int2 pa = pl[blockIdx.x];
   const int a = pa.x, top = pa.y;
   const int np = v.ann_np[a], c0 = v.ann_off[a];
   const int d = v.ann_disk[a];
   const DiskParams &P = v.dp[d];
   if( threadIdx.x == 0 ){
      double E = 0.0;
      for( int i=0 ; i<np ; ++i ) E += v.ctPole[c0 + i];
      s_E = E/np;
   }
   __syncthreads();
   const int j = v.ann_j[a];
   const double *rj = v.rj + P.rj0 + 1;
   const double dl = rj[j]-rj[j-1];                   /* z-face dl = dr */
   const double dt = v.ds[d].dt*v.dtfac;
   const R E = (R)s_E;
   const int *own = top ? v.consZR : v.consZL;
   for( int i=threadIdx.x ; i<np ; i+=blockDim.x ) v.fX[own[c0 + i]] = (double)E*dl*dt;
}

/* get_which4 (bfields.c:834-885): which of four phi edges is smallest (mode
 * 0) or largest (mode 1), comparing pairs with the periodic wrap of
 * phi_switch (:818-832), and the toggles of the two pairs not chosen */
__device__ __forceinline__ int ct_phi_switch(double dphi, double Pmax, int mode, int *err){
   int n = 0;
   while( dphi > .5*Pmax ){ dphi -= Pmax; if( ++n > WRAP_CAP ){ *err |= ERRF_WRAP; break; } }
   while( dphi <-.5*Pmax ){ dphi += Pmax; if( ++n > WRAP_CAP ){ *err |= ERRF_WRAP; break; } }
   if( mode == 1 ) dphi = -dphi;
   return dphi > 0. ? 1 : 0;
}
__device__ __forceinline__ int ct_which4(double phi, double phiR, double phiU, double phiUR,
                                         int *LR_alt, int *UD_alt, int mode, double Pmax, int *err){
   int LR_D = ct_phi_switch(phi - phiR, Pmax, mode, err);
   int LR_U = ct_phi_switch(phiU - phiUR, Pmax, mode, err);
   double phi1 = LR_D ? phiR : phi;
   double phi2 = LR_U ? phiUR : phiU;
   int UD = ct_phi_switch(phi1 - phi2, Pmax, mode, err);
   int which4 = UD == 0 ? (LR_D == 0 ? 0 : 1) : (LR_U == 0 ? 2 : 3);
   if( mode == 0 ){
      *LR_alt = (which4 == 0 || which4 == 1) ? LR_U : LR_D;
      if( which4 == 0 || which4 == 2 ) *UD_alt = ct_phi_switch(phiR - phiUR, Pmax, mode, err);
      else                             *UD_alt = ct_phi_switch(phi - phiU, Pmax, mode, err);
   }
   return which4;
}

/* E_phi of the face cell c owns on side s (0 inner r, 1 outer r, 2 lower z,
 * 3 upper z), as riemann_trans left it (riemann.c:188-212); cell (jc, kc) */
template<class R>
__device__ __forceinline__ R ct_ephi(const ViewT<R> &v, const DiskParams &P, int c, int jc,
                                     int kc, int s){
   int t, f;
   if( s == 0 ){ t = P.trr0 + (jc-1) + (P.Nr-1)*kc; f = v.consR[c]; }
   else if( s == 1 ){ t = P.trr0 + jc + (P.Nr-1)*kc; f = v.consL[c]; }
   else if( s == 2 ){ t = P.trz0 + jc + P.Nr*(kc-1); f = v.consZR[c]; }
   else { t = P.trz0 + jc + P.Nr*kc; f = v.consZL[c]; }
   return v.tr_flux[t] ? v.fEphi[f] : R(0.0);
}

/* make_edge_adjust, one thread per cell, which is list M (0..3) of the four
 * lines it borders: the line (jl, kl) is the r_jph[jl], z_kph[kl] edge; its
 * lists are the annuli (jl,kl) [c], (jl+1,kl) [cR], (jl,kl+1) [cU],
 * (jl+1,kl+1) [cUR], each from its I0, and the reference merges them by
 * repeated get_which4, ties to the lower list index.  A cell of list M at
 * position t is consumed at step e = t + (cells of each other list before
 * it): two of those counts are the cell's position in the face list of the
 * track it shares with that list minus t, the third (the diagonal annulus) a
 * binary search.
 *
 * The step's rank is stored at the two faces the cell ends there (frk: for
 * an r face the line below it in slot 0, above it in slot 1; for a z face
 * the line inside / outside it), where k_ct_update reads it beside its
 * neighbours.  Instruction-bound: the lists are numbered at compile time
 * (indexed at run time, the counts and cells lay in local memory and each
 * step branched four ways on the list consumed), and the 3 x 3 annuli around
 * the block are read once, into shared memory. */
struct LineAnn { int off, np, I0; };

template<int M, class R>
__device__ __forceinline__ void ct_line_step(const ViewT<R> &v, const DiskParams &P, const LineAnn (*A)[3],
                                             const int *f4, const int *o4, int c, int j, int k, int t, int np,
                                             double ux, double dt, int *err){
   const int jl = j - (M & 1), kl = k - (M >> 1);
   if( jl < 0 || jl > P.Nr-2 || kl < 0 || kl > P.Nz-2 ) return;
   const double Pmax = P.Pmax;
   /* the cell's r and z face of this line (0 inner r, 1 outer r, 2 lower z,
    * 3 upper z), and the counts their lists give */
   constexpr int sr = (M & 1) ? 0 : 1, sz = (M >> 1) ? 2 : 3;
   const int fr = f4[sr], fz = f4[sz];
   /* list n's annulus, relative to the cell's */
   auto ann = [&](int n) -> const LineAnn & { return A[1 + (n >> 1) - (M >> 1)][1 + (n & 1) - (M & 1)]; };
   int cnt[4];
   cnt[M] = t;
   cnt[M ^ 1] = fr - o4[sr] - t;
   cnt[M ^ 2] = fz - o4[sz] - t;
   {                                /* diagonal: cells of list n before this one */
      constexpr int n = M ^ 3;
      const LineAnn a = ann(n);
      /* both lists unrolled from I0: the count is near t nn / np */
      cnt[n] = gallop_lb(0, a.np, __float2int_rz(__fdividef((float)t*(float)a.np, (float)np)), [&](int mid){
         int s = a.I0 + mid; if( s >= a.np ) s -= a.np;
         double uy = v.piph[a.off + s];
         return !(n < M ? uy <= ux : uy < ux);
      });
   }
   const int e = cnt[0] + cnt[1] + cnt[2] + cnt[3];
   const int line = P.ln0 + jl + (P.Nr-1)*kl;
   const int l0 = v.line_off[line];
   if( e < 0 || e >= v.line_off[line+1] - l0 ){ *err |= ERRF_INTERNAL; return; }
   const size_t Nf = v.Nf;
   v.frk[(M >> 1) ? fr : Nf + fr] = e;
   v.frk[(M & 1) ? fz : Nf + fz] = e;
   /* the reference's state at step e */
   int cur[4];
   bool bad = false;
#pragma unroll
   for( int n=0 ; n<4 ; ++n ){
      if( n == M ){ cur[n] = c; continue; }
      const LineAnn a = ann(n);
      int s = a.I0 + cnt[n];                 /* I0 < np, 0 <= cnt <= np */
      if( s >= a.np ) s -= a.np;
      if( s < 0 || s >= a.np ){ bad = true; s = 0; }
      cur[n] = a.off + s;
   }
   if( bad ){ *err |= ERRF_INTERNAL; return; }
   double xp[4], xm[4];
#pragma unroll
   for( int n=0 ; n<4 ; ++n ){ xp[n] = n == M ? ux : v.piph[cur[n]]; xm[n] = xp[n] - v.dphi[cur[n]]; }
   int LR_alt = 0, UD_alt = 0;
   const int w4 = ct_which4(xp[0], xp[1], xp[2], xp[3], &LR_alt, &UD_alt, 0, Pmax, err);
   const int w4b = ct_which4(xm[0], xm[1], xm[2], xm[3], NULL, NULL, 1, Pmax, err);
   if( w4 != M ) *err |= ERRF_INTERNAL;
   /* E_phi of the cells' owned faces: c [3],[1]; cR [3],[0]; cU [1],[2];
    * cUR [0],[2]: the cell's own two, and one of the other row's and of the
    * other column's each */
   auto eph = [&](int n, int s){ return ct_ephi(v, P, cur[n], jl + (n & 1), kl + (n >> 1), s); };
   auto own = [&](int s, int f){
      const int tr = s <= 1 ? P.trr0 + jl + (P.Nr-1)*k : P.trz0 + j + P.Nr*kl;
      return v.tr_flux[tr] ? v.fEphi[f] : R(0.0);
   };
   const R q4 = R(.25);
   R E = q4*( own(sz, fz) + own(sr, fr) );
   if( M < 2 ){ if( LR_alt == 0 ) E += q4*eph(2,1); else E += q4*eph(3,0); }
   else       { if( LR_alt == 0 ) E += q4*eph(0,1); else E += q4*eph(1,0); }
   if( (M & 1) == 0 ){ if( UD_alt == 0 ) E += q4*eph(1,3); else E += q4*eph(3,2); }
   else              { if( UD_alt == 0 ) E += q4*eph(0,3); else E += q4*eph(2,2); }
   const double xmb = w4b == 0 ? xm[0] : w4b == 1 ? xm[1] : w4b == 2 ? xm[2] : xm[3];
   const double *rj = v.rj + P.rj0 + 1;
   double dl = (.5*(rj[jl]+rj[jl]))*get_dp(ux, xmb, Pmax, err);     /* get_dL(.,.,0) */
   v.lineX[l0 + e] = (double)E*dl*dt;
}

template<class R>
__global__ void __launch_bounds__(CB, MB_CT_LINE) k_ct_line(ViewT<R> v){
   __shared__ LineAnn A[3][3];
   __shared__ int s_o[4];
   const CellBlk b = v.cblk[blockIdx.x];
   const int i = b.y + threadIdx.x, np = b.np, j = b.j, k = b.k;
   const DiskParams &P = v.dp[b.disk];
   if( P.Nz < 2 ) return;
   if( threadIdx.x < 9 ){
      const int dk = (int)threadIdx.x/3, dj = (int)threadIdx.x%3, jj = j + dj - 1, kk = k + dk - 1;
      if( jj >= 0 && jj < P.Nr && kk >= 0 && kk < P.Nz ){
         const int a = P.ann0 + jj + P.Nr*kk;
         A[dk][dj] = {v.ann_off[a], v.ann_np[a], v.I0[a]};
      }
   }else if( threadIdx.x >= 32 && threadIdx.x < 36 ){  /* first faces of the annulus's four tracks */
      const int s = threadIdx.x - 32;
      int tr = -1;
      if( s == 0 && j >= 1 )      tr = P.trr0 + (j-1) + (P.Nr-1)*k;
      if( s == 1 && j <= P.Nr-2 ) tr = P.trr0 + j + (P.Nr-1)*k;
      if( s == 2 && k >= 1 )      tr = P.trz0 + j + P.Nr*(k-1);
      if( s == 3 && k <= P.Nz-2 ) tr = P.trz0 + j + P.Nr*k;
      s_o[s] = tr >= 0 ? v.tr_off[tr] : 0;
   }
   __syncthreads();
   if( i >= np ) return;
   const int c = b.c0 + i;
   const double dt = v.ds[b.disk].dt*v.dtfac;
   int err = 0;
   int t = i - A[1][1].I0;
   if( t < 0 ) t += np;
   const double ux = v.piph[c];
   const int f4[4] = {v.consR[c], v.consL[c], v.consZR[c], v.consZL[c]};
   const int o4[4] = {s_o[0], s_o[1], s_o[2], s_o[3]};
   ct_line_step<0,R>(v, P, A, f4, o4, c, j, k, t, np, ux, dt, &err);
   ct_line_step<1,R>(v, P, A, f4, o4, c, j, k, t, np, ux, dt, &err);
   ct_line_step<2,R>(v, P, A, f4, o4, c, j, k, t, np, ux, dt, &err);
   ct_line_step<3,R>(v, P, A, f4, o4, c, j, k, t, np, ux, dt, &err);
   raise_err(v, err);
}

/* The edge steps of line l that fall on face f of a track: the steps whose
 * pointer sum over the face's pair of lists equals the face's index d, i.e.
 * after the element that ends face d-1 up to the one that ends face d; face
 * 0 also takes the steps after the pair's last element (the pair has
 * wrapped).  slot: which of the face's two lines l is (frk).  Applied in
 * step order as S += sign X. */
template<class R>
__device__ __forceinline__ double ct_line_terms(const ViewT<R> &v, double S, int line, int tr,
                                                int f, int slot, double sign){
   const int l0 = v.line_off[line], ne = v.line_off[line+1] - l0;
   const double *X = v.lineX + l0;
   const int *frk = v.frk + (size_t)slot*v.Nf;
   /* a face whose rank k_ct_line did not store (positions that are not finite,
    * flagged there) holds anything */
   auto rank = [&](int g){ const int e = frk[g]; return (unsigned)e < (unsigned)ne ? e : 0; };
   int f0 = v.tr_off[tr], f1 = v.tr_off[tr+1];
   int hi = rank(f);
   int lo = f == f0 ? 0 : rank(f-1) + 1;
   for( int e=lo ; e<=hi ; ++e ) S += sign*X[e];
   if( f == f0 ) for( int e=rank(f1-1)+1 ; e<ne ; ++e ) S += sign*X[e];
   return S;
}

/* update_B_fluxes on the slots of cell c (r part, then z part, then
 * make_edge_adjust), then (first substep) move_cells / clean_pi / calc_dp
 * as k_update does without CT */
template<class R>
__global__ void __launch_bounds__(CB, MB_CT_UPDATE) k_ct_update(ViewT<R> v, int first){
   const CellBlk b = v.cblk[blockIdx.x];
   int a = b.x, i = b.y + threadIdx.x;
   int np = b.np;
   if( i >= np ) return;
   int c0 = b.c0, c = c0 + i;
   const DiskParams &P = v.dp[b.disk];
   int j = b.j, k = b.k;
   const double *X = v.fX;
   const bool z3 = v.ct == 2 && P.Nz > 1;
   /* own face f (the track's first face o) and the face before it */
   auto fm_of = [&](int f, int tr){ return f > v.tr_off[tr] ? f-1 : v.tr_off[tr+1]-1; };
   /* the RK snapshot / average of the slots (timestep.c:22, adjust_RK_cons
    * misc.c:239-241), taken here as their one read before the update */
   double st[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
   if( z3 ) rk_start<5>(v.Phi, v.RKPhi, v.nfs, c, first, st);
   else     rk_start<3>(v.Phi, v.RKPhi, v.nfs, c, first, st);
   double P0 = st[0], S1 = st[1], S2 = st[2], S3 = st[3], S4 = st[4];
   int f1 = -1, f2 = -1, f3 = -1, f4 = -1, t1 = 0, t2 = 0, t3 = 0, t4 = 0;
   if( j >= 1 ){                           /* inner r face: owned with LRtype 1 */
      t1 = P.trr0 + (j-1) + (P.Nr-1)*k;
      f1 = v.consR[c];
      int fm = fm_of(f1, t1);
      P0 = P0 - X[f1];
      S1 = f1 > v.tr_off[t1] ? (S1 + X[fm]) - X[f1] : (S1 - X[f1]) + X[fm];
   }
   if( j <= P.Nr-2 ){                      /* outer r face: LRtype 0 */
      t2 = P.trr0 + j + (P.Nr-1)*k;
      f2 = v.consL[c];
      int fm = fm_of(f2, t2);
      P0 = P0 + X[f2];
      S2 = f2 > v.tr_off[t2] ? (S2 + X[fm]) - X[f2] : (S2 - X[f2]) + X[fm];
   }
   if( z3 ){
      if( k >= 1 ){                        /* lower z face: LRtype 1, R->Phi[3] += X */
         t3 = P.trz0 + j + P.Nr*(k-1);
         f3 = v.consZR[c];
         int fm = fm_of(f3, t3);
         P0 = P0 + X[f3];
         S3 = f3 > v.tr_off[t3] ? (S3 - X[fm]) + X[f3] : (S3 + X[f3]) - X[fm];
      }
      if( k <= P.Nz-2 ){                   /* upper z face: LRtype 0, L->Phi[4] += X */
         t4 = P.trz0 + j + P.Nr*k;
         f4 = v.consZL[c];
         int fm = fm_of(f4, t4);
         P0 = P0 - X[f4];
         S4 = f4 > v.tr_off[t4] ? (S4 - X[fm]) + X[f4] : (S4 + X[f4]) - X[fm];
      }
      /* make_edge_adjust: lines in (k, j) order; add_E_phi takes L -, R +,
       * U -, D + (bfields.c:384-389) */
      const int ln = P.ln0;
      const int W = P.Nr-1;
      if( f2 >= 0 ){                       /* r face (j, j+1) at layer k */
         if( k >= 1 )      S2 = ct_line_terms(v, S2, ln + j + W*(k-1), t2, f2, 0, -1.0);
         if( k <= P.Nz-2 ) S2 = ct_line_terms(v, S2, ln + j + W*k, t2, f2, 1, 1.0);
      }
      if( f1 >= 0 ){                       /* r face (j-1, j) at layer k */
         if( k >= 1 )      S1 = ct_line_terms(v, S1, ln + (j-1) + W*(k-1), t1, f1, 0, -1.0);
         if( k <= P.Nz-2 ) S1 = ct_line_terms(v, S1, ln + (j-1) + W*k, t1, f1, 1, 1.0);
      }
      if( f4 >= 0 ){                       /* z face (k, k+1) of column j */
         if( j >= 1 )      S4 = ct_line_terms(v, S4, ln + (j-1) + W*k, t4, f4, 0, 1.0);
         if( j <= P.Nr-2 ) S4 = ct_line_terms(v, S4, ln + j + W*k, t4, f4, 1, -1.0);
      }
      if( f3 >= 0 ){                       /* z face (k-1, k) of column j */
         if( j >= 1 )      S3 = ct_line_terms(v, S3, ln + (j-1) + W*(k-1), t3, f3, 0, 1.0);
         if( j <= P.Nr-2 ) S3 = ct_line_terms(v, S3, ln + j + W*(k-1), t3, f3, 1, -1.0);
      }
      v.Phi[AT_PHI(3, c)] = S3;
      v.Phi[AT_PHI(4, c)] = S4;
      if( !first && f3 >= 0 ) v.fPhi[f3] = S3;
      if( !first && f4 >= 0 ) v.fPhi[f4] = S4;
   }
   v.Phi[AT_PHI(1, c)] = S1;
   v.Phi[AT_PHI(2, c)] = S2;
   v.Phi[AT_PHI(0, c)] = P0;
   if( !first && f1 >= 0 ) v.fPhi[f1] = S1;
   if( !first && f2 >= 0 ) v.fPhi[f2] = S2;
   if( first ){
      int err = 0;
      int cprev = c0 + (i == 0 ? np-1 : i-1);
      double piph = v.piph_new[c];
      v.dphi[c] = get_dp(piph, v.piph_new[cprev], P.Pmax, &err);
      v.piph[c] = piph;
      raise_err(v, err);
   }
}

/* check_flipped: face g is flagged when its owner's piph now lies before
 * the previous face's owner's (r and z tracks) */
template<class R>
__global__ void __launch_bounds__(FB) k_ct_flag(ViewT<R> v){
   const FaceBlk b = v.fblk[blockIdx.x];
   int t = b.x;
   if( b.dim == 2 && v.ct != 2 ) return;
   int f = b.f0 + b.y + threadIdx.x;
   if( f >= b.f1 ) return;
   const DiskParams &P = v.dp[b.disk];
   int err = 0;
   int fm = f > b.f0 ? f-1 : b.f1-1;
   int own = v.fLR[f] == 0 ? v.fL[f] : v.fR[f];
   int ownm = v.fLR[fm] == 0 ? v.fL[fm] : v.fR[fm];
   double dp = get_signed_dp(v.piph[own], v.piph[ownm], P.Pmax, &err);
   v.fFlip[f] = dp < 0. ? 1 : 0;
   raise_err(v, err);
}

/* flip_fluxes, one warp per track */
template<class R>
__global__ void k_ct_flip(ViewT<R> v){
   int t = (blockIdx.x*blockDim.x + threadIdx.x) >> 5;
   int lane = threadIdx.x & 31;
   if( t >= v.Ntr ) return;
   bool zf = v.tr_dim[t] == 2;
   if( zf && v.ct != 2 ) return;
   int o = v.tr_off[t], n = v.tr_off[t+1] - o;
   for( int base=0 ; base<n ; base+=32 ){
      bool fl = base + lane < n && v.fFlip[o + base + lane];
      unsigned m = __ballot_sync(0xffffffffu, fl);
      if( lane == 0 ){
         while( m ){
            int f = o + base + __ffs(m) - 1;
            m &= m - 1;
            int fm = f > o ? f-1 : o+n-1;
            int fp = f < o+n-1 ? f+1 : o;
            double *Pf = ct_slot(v, v.Phi, f, zf), *Rf = ct_slot(v, v.RKPhi, f, zf);
            double *Pm = ct_slot(v, v.Phi, fm, zf), *Rm = ct_slot(v, v.RKPhi, fm, zf);
            double *Pp = ct_slot(v, v.Phi, fp, zf), *Rp = ct_slot(v, v.RKPhi, fp, zf);
            double ph = *Pf, rk = *Rf;
            *Pf = *Pm + ph;
            *Rf = *Rm + rk;
            *Pm = -ph;
            *Rm = -rk;
            *Pp = *Pp + ph;
            *Rp = *Rp + rk;
            v.fLR[f] ^= 1;
            v.fLR[fm] ^= 1;
         }
      }
      __syncwarp();
   }
}

/* B_faces_to_cells type 1 for a real cell (bfields.c:88-309): cons[BRR]
 * (cons[BZZ]) from the fluxes of the cell's r (z) faces -- inner / lower
 * track first, each in face order -- over their
 * area, cons[BPP] from the two phi faces, with the moved cell's volume */
template<class R, bool FACE>
__device__ void ct_cons_B(const ViewT<R> &v, const DiskParams &P, int a, int c0, int np, int i,
                          int j, int k, double rp, double rm, double zp, double zm, double *cons,
                          int *err){
   int c = c0 + i, cm = c0 + (i == 0 ? np-1 : i-1);
   int I0 = v.I0[a];
   double S = 0.0, T = 0.0;
   double Sz = 0.0, Tz = 0.0;
   const bool z3 = v.ct == 2 && P.Nz > 1;
   const int tri = P.trr0 + (j-1) + (P.Nr-1)*k, tro = P.trr0 + j + (P.Nr-1)*k;
   const int tzi = P.trz0 + j + P.Nr*(k-1), tzo = P.trz0 + j + P.Nr*k;
   if( FACE && v.topo_set ){
      /* no flips since k_ct_update (the second substep): the fluxes face by
       * face (fPhi), a run being two streams of consecutive loads */
      auto sum = [&](int f){ S += v.fPhi[f]; T += v.fdA[f]; };
      auto zsum = [&](int f){ Sz += v.fPhi[f]; Tz += v.fdA[f]; };
      if( j >= 1 )      ct_over_runs(v, v.consR, tri, c0, np, i, I0, sum);
      if( j <= P.Nr-2 ) ct_over_runs(v, v.consL, tro, c0, np, i, I0, sum);
      if( z3 && k >= 1 )      ct_over_runs(v, v.consZR, tzi, c0, np, i, I0, zsum);
      if( z3 && k <= P.Nz-2 ) ct_over_runs(v, v.consZL, tzo, c0, np, i, I0, zsum);
   }else{
      /* through the slot of each face's owner by its LRtype, which flips may
       * have toggled (several faces can name one slot then): every face of
       * the cell's run in its inner (lower) track has the cell as R, in its
       * outer (upper) track as L; the other side's cell is read only when
       * that one owns the face */
      auto sum_in = [&](int f){ S += v.fLR[f] == 0 ? v.Phi[AT_PHI(2, v.fL[f])] : v.Phi[AT_PHI(1, c)]; T += v.fdA[f]; };
      auto sum_out = [&](int f){ S += v.fLR[f] == 0 ? v.Phi[AT_PHI(2, c)] : v.Phi[AT_PHI(1, v.fR[f])]; T += v.fdA[f]; };
      auto sum_zin = [&](int f){ Sz += v.fLR[f] == 0 ? v.Phi[AT_PHI(4, v.fL[f])] : v.Phi[AT_PHI(3, c)]; Tz += v.fdA[f]; };
      auto sum_zout = [&](int f){ Sz += v.fLR[f] == 0 ? v.Phi[AT_PHI(4, c)] : v.Phi[AT_PHI(3, v.fR[f])]; Tz += v.fdA[f]; };
      if( j >= 1 )      ct_over_runs(v, v.consR, tri, c0, np, i, I0, sum_in);
      if( j <= P.Nr-2 ) ct_over_runs(v, v.consL, tro, c0, np, i, I0, sum_out);
      if( z3 && k >= 1 )      ct_over_runs(v, v.consZR, tzi, c0, np, i, I0, sum_zin);
      if( z3 && k <= P.Nz-2 ) ct_over_runs(v, v.consZL, tzo, c0, np, i, I0, sum_zout);
   }
   double x0 = v.ann_rc[a];                          /* centroid_r(rp, rm) */
   double dph = get_dp(v.piph[c], v.piph[cm], P.Pmax, err);
   double dV = dV_of(rp, rm, dph, zp, zm);
   double dA = (rp-rm)*(zp-zm);
   double rfac = 1.0/x0;                                /* bfield_scale_factor(x0, 0) */
   double hr = 1.0, hp = x0;
   cons[BRR] = S * (dV*rfac/(T * hr));
   cons[BPP] = .5*(v.Phi[AT_PHI(0, c)]+v.Phi[AT_PHI(0, cm)])*dV/(dA * hp);
   if( z3 ){
      double zfac = 1.0, hz = 1.0;                      /* bfield_scale_factor(x2, 2) */
      cons[BZZ] = Sz * (dV*zfac/(Tz * hz));
   }
}

/* set_B_fields (bfields.c:44-80): each r (z) face's flux prim[BRR] dA
 * (prim[BZZ] dA) at its centre, into its owner's slot */
template<int Q, int NC, class R>
__global__ void __launch_bounds__(FB) k_ct_face_init(ViewT<R> v){
   const FaceBlk b = v.fblk[blockIdx.x];
   int t = b.x;
   bool zf = b.dim == 2;
   if( zf && v.ct != 2 ) return;
   int f = b.f0 + b.y + threadIdx.x;
   if( f >= b.f1 ) return;
   const DiskParams &P = v.dp[b.disk];
   int j = b.j, k = b.k;
   const double *rj = v.rj + P.rj0 + 1;
   const double *zk = v.zk + P.zk0 + 1;
   double prim[Q];
   if( !zf ){
      double x[3] = { .5*(rj[j]+rj[j]), v.fphic[f], 0.5*(zk[k]+zk[k-1]) };
      initial<Q,NC>(P, prim, x);
      *ct_slot(v, v.Phi, f, false) = prim[BRR]*v.fdA[f];
   }else{
      double x[3] = { centroid_r(rj[j], rj[j-1]), v.fphic[f], .5*(zk[k]+zk[k]) };
      initial<Q,NC>(P, prim, x);
      *ct_slot(v, v.Phi, f, true) = prim[BZZ]*v.fdA[f];
   }
}

}  // namespace disco

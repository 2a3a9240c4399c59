// shdom_grad.cuh -- Levis approximate gradient on the GPU (included by
// shdom_gpu.cu after the render kernel, whose traversal it shares).
//
// LEVISAPPROX_GRADIENT, adjoint branch (src/polarized/shdomsub4.f:288-809):
// with the radiance field frozen, the derivative of a weighted sum of
// rendered radiances, sum_r w_r I_r, with respect to the extinction and
// single-scattering albedo of one species on the property grid is
//  (i)  the derivative of the local source x extinction at the grid points
//       a ray visits (GRAD8 of COMPUTE_SOURCE_GRAD_1CELL, :1546-2042),
//       integrated along the ray with the ray's transmission;
//  (ii) the change of the ray's own attenuation, weighted by the radiance
//       still to come from beyond each path interval
//       (COMPUTE_RADIANCE_DERIVATIVE_ADJOINT, :4037-4114);
//  (iii) the change of the direct solar beam at the points whose exact
//       single scattering (and surface reflection) the ray sees
//       (COMPUTE_DIRECT_BEAM_DERIV_ADJOINT, :4117-4143, with the sun-path
//       derivatives of DIRECT_BEAM_AND_PATHS_PROP, src/shdomsub5.f:1608-2345).
//
// Four rays per warp, eight lanes each, one corner of the ray's cell per lane;
// a lane keeps its corner's source and source gradient while the ray's next
// cells share it.  Instead of storing the path (the reference's
// PASSED* arrays) the ray is traversed twice: pass A sums the radiance
// contributions F_n, pass B recomputes them in the same order and gets the
// radiance still to come at interval n as (R - sum_{k<n} F_k) / T_n with an
// FP64 running sum.  Within a cell every interval's contribution to a
// corner is a scalar weight times that corner's GRAD8, so the FP64 atomics
// into the gradient are issued once per cell.
#pragma once

namespace shdom {

struct GradArgs {
  RenderArgs r;
  const float *radiance;                   // [npts][nlm]
  const int *nr;                           // radiance truncation per point
  const int *interpptr;                    // [npts][8] property point of each trilinear corner
  const float *optinterpwt;                // [npts][8]
  const float *planck;                     // thermal source: [npts] B(T) of each point, else null
  const float *dextm;                      // [ng][2] delta-M scaled d(extinction)/d(unknown)
  const float *dalbm, *dfj;                // [npts][8][2]
  const float *alb_sp;                     // [npts] scaled albedo of the species
  const int *sj_ptr, *sj_iph;              // CSR per point: mixed exact single scatter of the species
  const float *sj_w;
  const float *legent_u;                   // [npts][nl] species phase series, unscaled
  const float *legent_s;                   // [npts][nl] property-mixed, delta-M scaled (several species)
  const float *fmix;                       // [npts] (several species)
  const float *scatterj;                   // [npts]
  const float *legenp_u;                   // [ng][nl] unscaled phase series per property point
  const float *extp, *albp;                // [ng] species extinction and albedo
  const int *piph;                         // [ng][maxnmicro]
  const float *pphw;
  const double *adj;                       // [nrays] adjoint weight of each ray
  double *gradout;                         // [ng][2]
  double *beam;                            // [npts]
  const float *botalb;                     // surface albedo of the bottom points
  const uint8_t *cellflip;                 // [ncells] parities of each cell's low corner (k_cell_flip)
  int npart, maxnmicro, ng;
  float scatmin;
};

constexpr int GWARPS = 4;
constexpr int GRAYS = 4;   // rays per warp, eight lanes each

// Exact single scatter of phase function iph at this ray's scattering angle.
__device__ __forceinline__ float ss_phase(const RenderArgs &a, int sj, float sf, int iph) {
  return (1.f - sf) * a.phasetab[(size_t)sj * a.numphase + iph] + sf * a.phasetab[(size_t)(sj + 1) * a.numphase + iph];
}

// Two sums over the eight lanes of a ray (every lane of the warp takes
// part): after the first exchange the even lanes carry p and the odd ones q,
// which halves the FP64 additions.
__device__ __forceinline__ void ray_sum2(double p, double q, double &sp, double &sq) {
  const bool odd = threadIdx.x & 1;
  double v = odd ? q : p;
  v += __shfl_xor_sync(0xffffffffu, odd ? p : q, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  const double o = __shfl_xor_sync(0xffffffffu, v, 1);
  sp = odd ? o : v;
  sq = odd ? v : o;
}

// Where a ray enters the grid, its direction and its single-scatter table position.
struct LevisRay {
  double x, y, z, c[3], ci[3], adj;
  float mu, sf;
  int cell, sj;  // cell < 0: nothing to traverse
};

__device__ LevisRay levis_ray(const GradArgs &G, int ray) {
  const RenderArgs &a = G.r;
  const double pi = 3.141592653589793;
  LevisRay r;
  r.cell = -1; r.sj = 0; r.sf = 0.f; r.mu = 0.f; r.adj = 0.0;
  for (int k = 0; k < 3; ++k) { r.c[k] = 0.0; r.ci[k] = 1e6; }
  r.x = r.y = r.z = 0.0;
  if (ray >= a.nrays) return r;
  r.adj = G.adj[ray];
  if (r.adj == 0.0) return r;
  double x0 = a.camx[ray], y0 = a.camy[ray], z0 = a.camz[ray];
  const double mu2 = a.cammu[ray], phi2 = a.camphi[ray], st = sqrt(1.0 - mu2 * mu2);
  double sn, cn;
  sincos(phi2 - pi, &sn, &cn);
  r.mu = (float)mu2;
  const float ztop = a.zgrid[a.nz - 1];
  if (z0 > ztop) {
    if (-mu2 >= 0.0) return r;
    const double d = (ztop - z0) / -mu2;
    x0 += d * st * cn;
    y0 += d * st * sn;
    z0 = ztop;
  } else if (z0 < a.zgrid[0]) {
    if ((threadIdx.x & 7) == 0) atomicCAS(a.err, ERR_NONE, ERR_RAY_BELOW);
    return r;
  }
  if (a.deltam) {
    double cosscat = (double)a.solarmu * mu2 + sqrt((1.0 - (double)a.solarmu * a.solarmu) * (1.0 - mu2 * mu2)) * cos((double)a.solaraz - phi2);
    cosscat = fmax(fmin(1.0, cosscat), -1.0);
    const float F = (float)((a.nscatangle - 1) * (acos(cosscat) / pi) + 1);
    const int J = min(a.nscatangle - 1, (int)F);
    r.sf = F - J; r.sj = J - 1;
  }
  r.c[0] = st * cn; r.c[1] = st * sn; r.c[2] = -mu2;
  for (int k = 0; k < 3; ++k)
    if (fabs(r.c[k]) > 1e-6) r.ci[k] = 1.0 / r.c[k]; else { r.c[k] = 0; r.ci[k] = 1e6; }
  r.cell = locate_cell(a, x0, y0, z0);
  r.x = x0; r.y = y0; r.z = z0;
  return r;
}

// What one lane keeps of its corner: source J in the ray's direction, its
// exact single scatter, and (GRAD) in gv the source gradient for the corner's
// eight property neighbours, [neighbour][unknown] at a stride of the block
// (COMPUTE_SOURCE_GRAD_1CELL).
template <bool GRAD>
__device__ void levis_corner(const GradArgs &G, const LevisRay &ray, int ip, const float *ydir, const float *tl, float &J,
                             float &ss, float *gv) {
  const RenderArgs &a = G.r;
  const int nl = a.ml + 1, ns = a.ns[ip];
  const float *S = a.source + (size_t)ip * a.nlm;
  float s = 0.f;
  if ((a.nlm & 3) == 0) {
    float s1 = 0.f, s2 = 0.f, s3 = 0.f;
    for (int j = 0; j < ns; j += 4) {  // terms past ns are stored as zero
      const float4 v = *reinterpret_cast<const float4 *>(S + j), y = *reinterpret_cast<const float4 *>(ydir + j);
      s = fmaf(v.x, y.x, s); s1 = fmaf(v.y, y.y, s1); s2 = fmaf(v.z, y.z, s2); s3 = fmaf(v.w, y.w, s3);
    }
    s = (s + s1) + (s2 + s3);
  } else {
    for (int j = 0; j < ns; ++j) s = fmaf(S[j], ydir[j], s);
  }
  // single scattering of the direct beam: with delta-M the exact term of
  // the unscaled phase function replaces the truncated one in the source;
  // without, the truncated term (from the series) is the single scatter
  const float dirf = a.dirflux[ip], da = dirf * a.secmu0;
  ss = 0.f;
  float sub = 0.f;
  if (ns > 0) {
    const float *cf = a.coef + (size_t)ip * a.nl;
    const int ls = a.lofj[ns - 1];
    for (int l = 0; l <= ls; ++l) sub += cf[l] * tl[l];
  }
  if (a.deltam) {
    s -= da * sub;
    float add = 0.f;
    for (int q = a.tms_ptr[ip]; q < a.tms_ptr[ip + 1]; ++q) add += a.tms_w[q] * ss_phase(a, ray.sj, ray.sf, a.tms_iph[q]);
    ss = da * add;
    s += ss;
  } else if (GRAD) {
    ss = da * sub;
  }
  J = s;
  if constexpr (GRAD) {
    float singscatj = 0.f;
    if (a.deltam)
      for (int q = G.sj_ptr[ip]; q < G.sj_ptr[ip + 1]; ++q) singscatj += G.sj_w[q] * ss_phase(a, ray.sj, ray.sf, G.sj_iph[q]);
    const float *lt = G.legent_u + (size_t)ip * nl;
    const float *Rp = a.nlm ? G.radiance + (size_t)ip * a.nlm : nullptr;
    const int rns = G.nr[ip];
    // sum_l f_l RY_l, RY_l = sum_m R(l, m) Ydir(l, m) over the point's
    // radiance terms, for the series of the point less one (d2), of a
    // property point less the point's (d1) and of the species (dj), each
    // with the direct beam's term added without delta-M
    const float beam = a.deltam ? 0.f : da;
    auto dots = [&](const float *lp, float &d1, float &d2, float &dj) {
      d1 = d2 = dj = 0.f;
      const float *ls = G.npart == 1 ? lt : G.legent_s + (size_t)ip * nl;
      for (int l = 0, j = 0; l < nl; ++l) {
        const int jn = j + 2 * min(l, a.mm) + 1;
        float ry = 0.f;
        for (; j < jn; ++j)
          if (j < rns) ry = fmaf(Rp[j], ydir[j], ry);
        const float t = ry + beam * tl[l], f = lt[l];
        d2 = fmaf(f - 1.f, t, d2);
        d1 = fmaf(lp[l] - f, t, d1);
        dj = fmaf(ls[l], t, dj);
      }
    };
    const float albip = G.alb_sp[ip];
    for (int nb = 0; nb < 8; ++nb) {
      float v[2] = {0.f, 0.f};
      const float xi = G.optinterpwt[(size_t)ip * 8 + nb];
      if (xi >= 1e-7f) {  // (one of the eight where the grid point is a property point)
        const int ib = G.interpptr[(size_t)ip * 8 + nb];
        float d1, d2, dj;
        dots(G.legenp_u + (size_t)ib * nl, d1, d2, dj);
        float sourcet;
        if (G.npart == 1) {
          sourcet = (albip > 1e-8f) ? s / albip : 0.f;
        } else {
          sourcet = 0.f;
          if (G.scatterj[ip] > G.scatmin) {
            sourcet = dj;
            if (a.deltam) sourcet += dirf * singscatj * a.secmu0 / (1.f - G.fmix[ip]);
          }
        }
        sourcet = fmaxf(0.f, sourcet);
        float ssp = 0.f;
        if (a.deltam)
          for (int q = 0; q < G.maxnmicro; ++q)
            ssp += G.pphw[(size_t)ib * G.maxnmicro + q] * ss_phase(a, ray.sj, ray.sf, G.piph[(size_t)ib * G.maxnmicro + q] - 1);
        const float ep = G.extp[ib], ap = G.albp[ib];
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const float DE = d == 0 ? 1.f : 0.f, DA = d == 1 ? 1.f : 0.f;
          const float DFJ = G.dfj[((size_t)ip * 8 + nb) * 2 + d], dal = G.dalbm[((size_t)ip * 8 + nb) * 2 + d];
          const float dex = G.dextm[(size_t)ib * 2 + d];
          const float dsource = (DE * ap + DA * ep) * d1 + DFJ * d2;
          v[d] = xi * (sourcet * (albip * dex + dal) + dsource);
          // emission e (1 - albedo) B (src/polarized/shdomsub4.f:2009-2016), no temperature unknowns
          if (G.planck) v[d] += xi * (G.planck[ip] * (1.f - albip) * dex - G.planck[ip] * dal);
          if (a.deltam) v[d] += dirf * a.secmu0 * xi * (singscatj * DFJ + DA * (ssp - singscatj) * ep + DE * (ssp - singscatj) * ap);
        }
      }
      gv[(2 * nb) * (GWARPS * 32)] = v[0];
      gv[(2 * nb + 1) * (GWARPS * 32)] = v[1];
    }
  }
}

// One pass over the rays of a warp (eight lanes each).  Returns the ray's
// radiance; with GRAD adds the gradient of adj times it, rtot the radiance of
// a first pass.
template <bool GRAD>
__device__ double levis_traverse(const GradArgs &G, const LevisRay &ray, const float *ydir, const float *tl, double rtot,
                                 float *gv) {
  const RenderArgs &a = G.r;
  const int lane = threadIdx.x & 31, k8 = lane & 7;
  const unsigned gmask = 0xffu << (lane & 24);
  const double cx = ray.c[0], cy = ray.c[1], cz = ray.c[2];
  const int bitx = cx < 0, bity = cy < 0, bitz = cz < 0, ioct0 = bitx + 2 * bity + 4 * bitz;
  const float xm = 0.5f * (a.xgrid[0] + a.xgrid[a.nx - 1]), ym = 0.5f * (a.ygrid[0] + a.ygrid[a.ny - 1]);
  const double eps = 1.0e-5 * (a.gridpos[3 * a.gridptr[7] + 2] - a.gridpos[3 * a.gridptr[0] + 2]);
  const double c12 = (double)0.08333333333f;
  double xe = ray.x, ye = ray.y, ze = ray.z;
  int cell = ray.cell;
  int mine = -1;  // the point this lane's J, ss and gradient are of
  float myJ = 0.f, myss = 0.f;
  double transmit = 1.0, cumf = 0.0, bound = 0.0;
  bool act = cell >= 0;
  int guard = 0;
  while (__any_sync(0xffffffffu, act)) {
    const int c = act ? cell : 0;
    // Lane k8 holds the corner whose grid indices have its parities (a cell
    // without width along an axis: its corner on that side), so a corner
    // shared with the next cell stays in its lane.
    const int cb = k8 ^ G.cellflip[c];
    const int *g = a.gridptr + 8 * (size_t)c;
    const int ip = g[cb];
    const float ext = a.text[ip];
    // a cell without extinction adds nothing and changes no transmission
    const unsigned cloudy = __ballot_sync(0xffffffffu, ext != 0.f);  // (every lane votes)
    const bool run = act && (cloudy & gmask);
    const float *P1 = a.gridpos + 3 * g[0], *P2 = a.gridpos + 3 * g[7];
    const float p1x = P1[0], p1y = P1[1], p1z = P1[2], p2x = P2[0], p2y = P2[1], p2z = P2[2];
    if (run && mine != ip) {
      levis_corner<GRAD>(G, ray, ip, ydir, tl, myJ, myss, gv);
      mine = ip;
    }
    __syncwarp();
    const int cf = a.cellflags[c];
    const bool ipinx = (cf & 1) && !((a.bcflag & 1) && ((cx > 0 && xe < xm) || (cx < 0 && xe > xm)));
    const bool ipiny = (cf & 2) && !((a.bcflag & 2) && ((cy > 0 && ye < ym) || (cy < 0 && ye > ym)));
    const double sox = ipinx ? 1e20 : ((bitx ? p1x : p2x) - xe) * ray.ci[0];
    const double soy = ipiny ? 1e20 : ((bity ? p1y : p2y) - ye) * ray.ci[1];
    const double soz = ((bitz ? p1z : p2z) - ze) * ray.ci[2];
    const double so = fmin(sox, fmin(soy, soz));
    if (act && so < -eps) { if (k8 == 0) atomicCAS(a.err, ERR_NONE, ERR_RAY_SO); act = false; }
    // Positions, path lengths, trilinear weights and the sums of weighted
    // corner values are FP64: the weight terms of the gradient are of the
    // size of the interpolated extinction, which cancels to nearly zero
    // beside clouds and in the extrapolating open-boundary edge cells.
    // Each lane forms the weight of its own corner only.
    if (__any_sync(0xffffffffu, run)) {
      const float delx = p2x - p1x, dely = p2y - p1y, delz = p2z - p1z;
      // one division for the three axes, an axis per lane
      const float del3 = k8 == 0 ? delx : k8 == 1 ? dely : delz;
      const double inv3 = k8 < 2 && del3 <= 0.f ? 1.0 : 1.0 / del3;
      const double idx = __shfl_sync(0xffffffffu, inv3, lane & 24), idy = __shfl_sync(0xffffffffu, inv3, (lane & 24) + 1),
                   idz = __shfl_sync(0xffffffffu, inv3, (lane & 24) + 2);
      const bool hx = cb & 1, hy = cb & 2, hz = cb & 4;
      // Rounded as the reference's: the position first, then its coordinate in
      // the cell.  Where a ray enters through one face and leaves through
      // another, the corner on neither has weight zero at both ends, and
      // whether that is exactly zero decides if the cell counts.
      const double u0 = (xe - p1x) * idx, v0 = (ye - p1y) * idy, q0 = (ze - p1z) * idz;
      const double un = (fma(so, cx, xe) - p1x) * idx, vn = (fma(so, cy, ye) - p1y) * idy, qn = (fma(so, cz, ze) - p1z) * idz;
      const double ux = hx ? u0 : 1 - u0, uy = hy ? v0 : 1 - v0, uz = hz ? q0 : 1 - q0;
      const double eD = run ? (double)ext : 0.0, jD = run ? (double)(myJ * ext) : 0.0;
      const double ss8 = (double)(myss * ext);  // this corner's single scatter x extinction
      double w1 = uz * uy * ux, e1, s1, en, sn;
      ray_sum2(w1 * eD, w1 * jD, e1, s1);
      const double wn = (hz ? qn : 1 - qn) * (hy ? vn : 1 - vn) * (hx ? un : 1 - un);
      ray_sum2(wn * eD, wn * jD, en, sn);
      s1 = fmax(0.0, s1);
      sn = fmax(0.0, sn);
      int ntau = 0;
      if (run) ntau = max(1, 1 + (int)(so * 0.5 * (e1 + en) / a.tautol));
      const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)ntau);
      const double dels = ntau > 1 ? so / ntau : so;
      // inside the cell the corner's weight is a product of lines in the path length
      double bx = 0.0, by = 0.0, bz = 0.0, step = 0.0;
      if (nmax > 1) {
        bx = cx * idx; by = cy * idy; bz = cz * idz;
        if (!hx) bx = -bx;
        if (!hy) by = -by;
        if (!hz) bz = -bz;
      }
      double accG = 0.0, accS = 0.0, accR = 0.0;  // per-cell weights of this lane's corner
      for (int it = 1; it <= nmax; ++it) {
        double w0 = wn, e0 = en, s0 = sn;
        if (it < nmax) {
          step += 1.0;
          const double sl = step * dels, wi = fma(sl, bz, uz) * fma(sl, by, uy) * fma(sl, bx, ux);
          double ei, si;
          ray_sum2(wi * eD, wi * jD, ei, si);
          if (it < ntau) { w0 = wi; e0 = ei; s0 = fmax(0.0, si); }
        }
        if (it <= ntau) {
          const double ex = 0.5 * (e0 + e1);
          if (ex != 0.0) {
            // abscell / ext = dels (1 - tau/2 (1 - tau/3)): no quotient by the extinction
            const double tau = ex * dels, poly = 1.0 - 0.5 * tau * (1.0 - 0.33333333333 * tau);
            const double transcell = 1.0 - tau * poly, dp = dels * poly;
            const double k = c12 * dels * (1.0 - 0.05 * (e1 - e0) * dels);
            // a field f of the interval contributes dp (0.5 (f0 + f1) + k (e0 f1 - e1 f0)) = c0 f0 + c1 f1
            const double c0 = dp * fma(-k, e1, 0.5), c1 = dp * fma(k, e0, 0.5);
            const double t0 = transmit * c0, t1 = transmit * c1;
            const double fn = fma(t0, s0, t1 * s1);
            if (GRAD) {
              const double wg = fma(t0, w0, t1 * w1);
              accG += wg;
              // the single scatter is interpolated with each corner's term
              // clamped at zero (SINGSCAT0/1 of ADJOINT_INTEGRATE_1RAY); the
              // trilinear weights go negative where open-boundary edge cells
              // extrapolate beyond the cell
              if ((__double2hiint(w0) | __double2hiint(w1) | __double2hiint(ss8)) < 0)
                accS += fma(t0, fmax(0.0, w0 * ss8), t1 * fmax(0.0, w1 * ss8));
              else
                accS = fma(ss8, wg, accS);
              // radiance still to come from the start (r1 / transmit) and from
              // the end of this interval (r0 / transmit)
              const double r1 = rtot - cumf, r0 = (r1 - fn) / transcell;
              accR += fma(c0 * r0, w0, c1 * r1 * w1);
            }
            cumf += fn;
            transmit *= transcell;
          } else {
            accS = 0.0;
          }
          e1 = e0; s1 = s0; w1 = w0;
        }
      }
      if (GRAD && run) {
        // source-gradient and attenuation terms of this lane's corner
        const double ag = ray.adj * accG, ar = -ray.adj * accR;
        if (ag != 0.0 || ar != 0.0) {
          const float4 *xw = reinterpret_cast<const float4 *>(G.optinterpwt + (size_t)ip * 8);
          const float4 xa = xw[0], xb = xw[1];
          const float xs[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
          for (int nb = 0; nb < 8; ++nb) {
            if (xs[nb] == 0.f) continue;
            const int ib = G.interpptr[(size_t)ip * 8 + nb];
            const float2 de = *reinterpret_cast<const float2 *>(G.dextm + (size_t)ib * 2);
            const double t0 = ag * (double)gv[(2 * nb) * (GWARPS * 32)] + (double)(de.x * xs[nb]) * ar;
            const double t1 = ag * (double)gv[(2 * nb + 1) * (GWARPS * 32)] + (double)(de.y * xs[nb]) * ar;
            if (t0 != 0.0) atomicAdd(&G.gradout[(size_t)ib * 2], t0);
            if (t1 != 0.0) atomicAdd(&G.gradout[(size_t)ib * 2 + 1], t1);
          }
        }
        const double bw = ray.adj * accS;
        if (bw != 0.0) atomicAdd(&G.beam[ip], bw);
      }
    }
    if (act) {
      int iface, jface;
      bool openbc;
      if (sox <= soz && sox <= soy) { iface = 1 - bitx; jface = 0; openbc = (cf & 1) && (a.bcflag & 1); }
      else if (soy <= soz) { iface = 3 - bity; jface = 1; openbc = (cf & 2) && (a.bcflag & 2); }
      else { iface = 5 - bitz; jface = 2; openbc = false; }
      const int nxt = a.neighptr[6 * (size_t)c + iface];
      int kface = iface, kc = c;
      if (openbc) { kface = iface ^ 1; kc = nxt; iface = -1; }
      double xn = xe + so * cx, yn = ye + so * cy, zn = ze + so * cz;
      if (nxt >= 0) {
        const float *q = a.gridpos + 3 * a.gridptr[8 * (size_t)nxt + ioct0];
        if (jface == 0) xn = q[0]; else if (jface == 1) yn = q[1]; else zn = q[2];
      }
      if (transmit < a.transcut) {
        act = false;
      } else if (nxt < 0 && iface >= 4) {
        act = false;
        const int *gk = a.gridptr + 8 * (size_t)kc;
        float xs[4], ys[4], rb[4], dr[4];
        int bp[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int q = gk[c_face[kface][k]];
          bp[k] = q; xs[k] = a.gridpos[3 * q]; ys[k] = a.gridpos[3 * q + 1]; dr[k] = 0.f;
          if (ray.mu < 0.f) rb[k] = a.skyrad;
          else {
            const int bi = a.bot_index[q];
            rb[k] = bi >= 0 ? a.bcrad_bot[bi] : 0.f;
            if (bi >= 0) dr[k] = 0.318309886f * G.botalb[bi] * a.dirflux[q];
          }
        }
        const double uu = (xs[1] - xs[0] > 0) ? (xn - xs[0]) / (xs[1] - xs[0]) : 0.0;
        const double vv = (ys[2] - ys[0] > 0) ? (yn - ys[0]) / (ys[2] - ys[0]) : 0.0;
        const double bi4[4] = {(1 - uu) * (1 - vv), uu * (1 - vv), (1 - uu) * vv, uu * vv};
        const float radbnd = (float)(bi4[0] * rb[0] + bi4[1] * rb[1] + bi4[2] * rb[2] + bi4[3] * rb[3]);
        bound = transmit * radbnd;
        if (GRAD) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k8 == k) {
              const double bw = ray.adj * transmit * bi4[k] * (double)dr[k];
              if (bw != 0.0) atomicAdd(&G.beam[bp[k]], bw);
            }
        }
      } else {
        cell = nxt;
        if (cell < 0 || ++guard >= (1 << 22)) act = false;
      }
      xe = xn; ye = yn; ze = zn;
    }
  }
  return cumf + bound;
}

// Per cell, which of its low corner's grid indices are odd (0 along an axis
// on which the cell has no width): bits x, y, z.
__global__ void k_cell_flip(const int *__restrict__ gridptr, int ncells, int ny1, int nz, uint8_t *__restrict__ flip) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const int lo = gridptr[8 * (size_t)c], hi = gridptr[8 * (size_t)c + 7];
  const int z0 = lo % nz, y0 = lo / nz % ny1, x0 = lo / nz / ny1, z1 = hi % nz, y1 = hi / nz % ny1, x1 = hi / nz / ny1;
  flip[c] = (uint8_t)((x0 != x1 ? x0 & 1 : 0) | (y0 != y1 ? (y0 & 1) << 1 : 0) | (z0 != z1 ? (z0 & 1) << 2 : 0));
}

// Pass A then pass B for the rays of a warp.  Dynamic shared memory: per ray
// the functions of its direction (nlm + 4 floats, so that the four rays of a
// warp read different banks) and t_l (32 floats).
//
// What bounds it: the FP64 pipe (68% busy; about 20 operations to cross an
// empty cell and 130 for a cloudy one).  So the ray scalars of an interval
// are two coefficients that every field and weight shares, the interior
// weights are products of lines, two sums share an exchange and the three
// axes a division.  Measured, 36864 rays through 64x64x32 with 20% cloud:
// 17.3 ms; without those 18.7; one warp per ray 142.
__global__ void __launch_bounds__(GWARPS * 32) k_levis_adjoint(GradArgs G) {
  extern __shared__ __align__(16) float gsm[];
  __shared__ float gvs[16 * GWARPS * 32];
  const RenderArgs &a = G.r;
  const int k8 = threadIdx.x & 7, lr = threadIdx.x >> 3;
  const int ystr = ((a.nlm + 3) & ~3) + 4;
  float *ydir = gsm + lr * ystr, *tl = gsm + GWARPS * GRAYS * ystr + lr * 32;
  const LevisRay ray = levis_ray(G, blockIdx.x * (GWARPS * GRAYS) + lr);
  if (ray.cell >= 0) {
    const int i = blockIdx.x * (GWARPS * GRAYS) + lr;
    ylm_dir_lanes(ydir, (float)a.cammu[i], (float)a.camphi[i], a.ml, a.mm, k8, 8);
  }
  __syncwarp();
  if (ray.cell >= 0)
    for (int l = k8; l <= a.ml; l += 8) {
      const int me = min(l, a.mm), j0 = (l <= a.mm) ? l * l : (2 * a.mm + 1) * l - a.mm * a.mm - a.mm;
      float s = 0.f;
      for (int k = 0; k < 2 * me + 1; ++k) s += ydir[j0 + k] * a.ylmsun[j0 + k];
      tl[l] = s;
    }
  __syncwarp();
  const double rtot = levis_traverse<false>(G, ray, ydir, tl, 0.0, nullptr);
  levis_traverse<true>(G, ray, ydir, tl, rtot, gvs + threadIdx.x);
}

// Direct-beam term: for each point with a non-zero beam weight, the sun
// path's d(optical path)/d(extinction) per property corner, cell by cell
// (the path of DIRECT_BEAM_PROP).  The weights are summed per property point
// (one atomic per corner); k_levis_beam_add turns the sums into both
// unknowns' derivatives.
struct BeamArgs {
  const float *gridpos, *zlev;
  const double *beam;
  double *sunpath;  // [ng] sum over points of beam weight times d(optical path)/d(extinction)
  int npts, npx, npy, npz, bcflag, ipflag;
  float delx, dely, solarmu, solaraz;
};

__global__ void k_levis_beam(BeamArgs b) {
  const int ipt = blockIdx.x * blockDim.x + threadIdx.x;
  if (ipt >= b.npts) return;
  const double weight = b.beam[ipt];
  if (weight == 0.0) return;
  const int npx = b.npx, npy = b.npy, npz = b.npz, bcflag = b.bcflag;
  int ipdirect = b.ipflag;
  if (b.ipflag & 4) ipdirect = 0;
  const double sunmu = -(double)b.solarmu, sunaz = (double)(float)(b.solaraz + 3.14159265f);
  double cx = sqrt(1.0 - sunmu * sunmu) * cos(sunaz), cy = sqrt(1.0 - sunmu * sunmu) * sin(sunaz);
  double cz = fabs(sunmu), cxinv, cyinv, czinv;
  if (fabs(cx) > 1e-6) cxinv = 1.0 / cx; else { cx = 0; cxinv = 1e20; }
  if (fabs(cy) > 1e-6) cyinv = 1.0 / cy; else { cy = 0; cyinv = 1e20; }
  if (fabs(cz) > 1e-6) czinv = 1.0 / cz; else { cz = 0; czinv = 1e20; }
  const int di = cx >= 0 ? 1 : -1, dj = cy >= 0 ? 1 : -1, dk = cz >= 0 ? 1 : -1;
  const double epsz = 1.0e-6 * (b.zlev[npz - 1] - b.zlev[0]);
  const double delxd = b.delx, delyd = b.dely, xdomain = delxd * npx, ydomain = delyd * npy;
  const double z = b.gridpos[3 * ipt + 2], x = b.gridpos[3 * ipt], y = b.gridpos[3 * ipt + 1];
  int il = 0, iu = npz;
  while (iu - il > 1) { int im = (iu + il) / 2; if (z >= b.zlev[im - 1]) il = im; else iu = im; }
  int k = max(il, 1);
  int i = (int)(x / delxd) + 1;
  if (i > npx && fabs(x - xdomain) < 0.001 * delxd) i = npx;
  int j = (int)(y / delyd) + 1;
  if (j > npy && fabs(y - ydomain) < 0.001 * delyd) j = npy;
  double xe = x, ye = y, ze = z, xp = xe, yp = ye, zp = ze;
  bool constx = ipdirect & 1, consty = ipdirect & 2;
  if (cx == 0.0) constx = true;
  if (cy == 0.0) consty = true;
  if ((bcflag & 1) && (fabs(x) < 0.01 * delxd || fabs(x - (npx - 1) * delxd) < 0.01 * delxd)) constx = true;
  if ((bcflag & 2) && (fabs(y) < 0.01 * delyd || fabs(y - (npy - 1) * delyd) < 0.01 * delyd)) consty = true;
  const int guard_max = 4 * (npx + npy + npz) * 64;
  for (int guard = 0; fabs(ze - b.zlev[npz - 1]) > epsz && guard < guard_max; ++guard) {
    int ipn = i + 1;
    if (i == npx) ipn = (bcflag & 1) ? npx : 1;
    int jpn = j + 1;
    if (j == npy) jpn = (bcflag & 2) ? npy : 1;
    const double x0 = delxd * (i - 1), x1 = x0 + delxd, y0 = delyd * (j - 1), y1 = y0 + delyd;
    const double z0 = b.zlev[k - 1], z1 = b.zlev[k];
    const int I1 = (k - 1) + npz * (j - 1) + npz * npy * (i - 1), I2 = (k - 1) + npz * (j - 1) + npz * npy * (ipn - 1);
    const int I3 = (k - 1) + npz * (jpn - 1) + npz * npy * (i - 1), I4 = (k - 1) + npz * (jpn - 1) + npz * npy * (ipn - 1);
    double sox, soy, soz;
    if (constx) sox = 1e30; else if (cx > 0) { sox = (x1 - xe) * cxinv; xp = x1; } else { sox = (x0 - xe) * cxinv; xp = x0; }
    if (consty) soy = 1e30; else if (cy > 0) { soy = (y1 - ye) * cyinv; yp = y1; } else { soy = (y0 - ye) * cyinv; yp = y0; }
    if (cz > 0) { soz = (z1 - ze) * czinv; zp = z1; } else if (cz < 0) { soz = (z0 - ze) * czinv; zp = z0; } else soz = 1e30;
    double xoffs = 0, yoffs = 0, so;
    if (soz <= sox && soz <= soy) {
      so = soz;
      if (!constx) xp = xe + so * cx;
      if (!consty) yp = ye + so * cy;
      k += dk;
    } else if (sox <= soy) {
      so = sox;
      if (!consty) yp = ye + so * cy;
      zp = ze + so * cz;
      i += di;
      if (i == 0) { if (bcflag & 1) { i = 1; constx = true; } else { i = npx; xoffs = xdomain; } }
      else if (i == npx + 1) { if (bcflag & 1) { i = npx; constx = true; } else { i = 1; xoffs = -xdomain; } }
    } else {
      so = soy;
      if (!constx) xp = xe + so * cx;
      zp = ze + so * cz;
      j += dj;
      if (j == 0) { if (bcflag & 2) { j = 1; consty = true; } else { j = npy; yoffs = ydomain; } }
      else if (j == npy + 1) { if (bcflag & 2) { j = npy; consty = true; } else { j = 1; yoffs = -ydomain; } }
    }
    so = fmax(so, 0.0);
    const double ax = 1.0 / (x1 - x0), ay = 1.0 / (y1 - y0), az = 1.0 / (z1 - z0);
    const double u0 = (xe - x0) * ax, v0 = (ye - y0) * ay, w0 = (ze - z0) * az;
    const double du = (xp - x0) * ax - u0, dv = (yp - y0) * ay - v0, dw = (zp - z0) * az - w0;
    // the path integral of each corner's trilinear weight: a cubic along the
    // segment, exact with the two-point Gauss rule
    constexpr double t1 = 0.21132486540518713, t2 = 0.78867513459481287;
    const double ua = fma(t1, du, u0), va = fma(t1, dv, v0), wa = fma(t1, dw, w0);
    const double ub = fma(t2, du, u0), vb = fma(t2, dv, v0), wb = fma(t2, dw, w0);
    const double h = 0.5 * so;
    const double a00 = (1 - va) * (1 - wa) * h, a10 = va * (1 - wa) * h, a01 = (1 - va) * wa * h, a11 = va * wa * h;
    const double b00 = (1 - vb) * (1 - wb) * h, b10 = vb * (1 - wb) * h, b01 = (1 - vb) * wb * h, b11 = vb * wb * h;
    const double path[8] = {(1 - ua) * a00 + (1 - ub) * b00, ua * a00 + ub * b00, (1 - ua) * a10 + (1 - ub) * b10, ua * a10 + ub * b10,
                            (1 - ua) * a01 + (1 - ub) * b01, ua * a01 + ub * b01, (1 - ua) * a11 + (1 - ub) * b11, ua * a11 + ub * b11};
    const int ptrs[8] = {I1, I2, I3, I4, I1 + 1, I2 + 1, I3 + 1, I4 + 1};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float dpath = (float)path[c];
      if (dpath != 0.f) atomicAdd(&b.sunpath[ptrs[c]], weight * dpath);
    }
    xe = xp + xoffs; ye = yp + yoffs; ze = zp;
  }
}

__global__ void k_levis_beam_add(const double *__restrict__ sunpath, const float *__restrict__ dextm, int ng, double *gradout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * ng) return;
  gradout[i] -= (double)dextm[i] * sunpath[i >> 1];
}

}  // namespace shdom

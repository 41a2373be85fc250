// CPU check of repr::vertex_point (tmc_gb300/csrc/dmc_repr.cuh): every contour it answers must get the
// floats of the float64 restatement of the reference.  Built with nvcc as host code.
//   point_check field.raw nx ny nz iso  -> prints "contours mismatches redone w64 excluded searched"
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../tmc_gb300/csrc/common.cuh"
#include "../../tmc_gb300/csrc/dmc_repr.cuh"

using namespace tmc;

static uint64_t polygon(unsigned cs, const float u[8], double iso) {
  if (!case_ambiguous(cs)) return table_contour(TMC_CASE_CONTOUR[cs]);
  uint64_t to = ~0ull;
  for (int f = 0; f < 6; f++) {
    const uint32_t fv = face_v_pack(f);
    const int fc = face_case(cs, fv);
    int sep = 0;
    if (fc == 6 || fc == 9) sep = decider(u[nib(fv, 0)], u[nib(fv, 1)], u[nib(fv, 2)], u[nib(fv, 3)]) >= iso;
    face_segments(fc, sep, face_e_pack(f), to);
  }
  return connect_contours(to, case_edge_mask(cs));
}

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const int nx = atoi(argv[2]), ny = atoi(argv[3]), nz = atoi(argv[4]);
  const double iso = atof(argv[5]);
  std::vector<float> f((size_t)nx * ny * nz);
  FILE* in = fopen(argv[1], "rb");
  if (!in || fread(f.data(), 4, f.size(), in) != f.size()) return 3;
  fclose(in);
  float iso_up = (float)iso;
  if ((double)iso_up < iso) iso_up = nextafterf(iso_up, INFINITY);
  long contours = 0, mism = 0, redone = 0, w64 = 0, excluded = 0, searched = 0;
  for (int k = 0; k < nz - 1; k++)
    for (int j = 0; j < ny - 1; j++)
      for (int i = 0; i < nx - 1; i++) {
        float u[8];
        for (int q = 0; q < 8; q++)
          u[q] = f[((size_t)(k + ((q >> 2) & 1)) * ny + (j + ((q >> 1) & 1))) * nx + i + (q & 1)];
        unsigned cs = 0;
        for (int q = 0; q < 8; q++) cs |= (unsigned)(u[q] >= iso_up) << q;
        if (cs == 0 || cs == 255) continue;
        const uint64_t c = polygon(cs, u, iso);
        const int n = cnt_count(c);
        repr::Boxes bx;
        float pts[4][36];
        uint32_t map = 0;
        for (int t = 0, flat = 0; t < n; flat += cnt_size(c, t++)) {
          for (int d = 0; d < 3; d++) { bx.b[t][d][0] = 1; bx.b[t][d][1] = 0; }
          for (int q = 0; q < cnt_size(c, t); q++) {
            const int e = cnt_edge(c, flat + q);
            map |= (uint32_t)t << (2 * e);
            float ui[3];
            repr::local_from_param(e, repr::edge_param_exact(e, u, iso), ui);
            for (int d = 0; d < 3; d++) {
              pts[t][3 * q + d] = ui[d];
              bx.b[t][d][0] = bx.b[t][d][0] > ui[d] ? ui[d] : bx.b[t][d][0];
              bx.b[t][d][1] = bx.b[t][d][1] < ui[d] ? ui[d] : bx.b[t][d][1];
            }
          }
        }
        const uint32_t crossed = repr::spread_edges(case_edge_mask(cs));
        for (int t = 0; t < n; t++) {
          contours++;
          const int sz = cnt_size(c, t);
          bool excl = false;
          for (int q = 0; q < n; q++) excl = excl || (sz != 3 && q != t && cnt_size(c, q) == 3);
          const uint32_t em = repr::edges_of_rank(map, t, crossed);
          // the whole search, as dmc_vertex_search_kernel runs it
          {
            float frame[repr::kFrameFloats];
            for (int q = 0; q < 8; q++) frame[q] = u[q];
            const repr::FrameCol F{frame, 1};
            const ffx::ff iso_ff = ffx::ff_from_double(iso);
            const bool exact_iso = (double)(float)iso == iso;
            repr::Exclusion X;
            bool ok = true;
            if (sz != 3)
              for (int q = 0; q < n; q++) {
                if (q == t || cnt_size(c, q) != 3) continue;
                ok = repr::contour_box(F, repr::edges_of_rank(map, q, crossed), iso, iso_ff, exact_iso, X.lo[X.n], X.hi[X.n]) && ok;
                for (int d = 0; d < 3; d++)
                  if (ok && (X.lo[X.n][d] != bx.b[q][d][0] || X.hi[X.n][d] != bx.b[q][d][1])) mism++;
                X.n++;
              }
            ffx::ff mean[3];
            auto mean64 = [&]() { return repr::mean_point_exact(pts[t], sz); };
            const int prj = ok ? repr::vertex_frame<true>(F, em, sz, iso, iso_ff, exact_iso, mean, mean64) : -1;
            if (prj >= 0) {
              const int ax[3][3] = {{0, 1, 2}, {0, 2, 1}, {1, 2, 0}};
              repr::Exclusion Y = X;
              for (int b = 0; b < X.n; b++)
                for (int d = 0; d < 3; d++) {
                  Y.lo[b][d] = X.lo[b][ax[prj][d]];
                  Y.hi[b][d] = X.hi[b][ax[prj][d]];
                }
              float p[3] = {0, 0, 0};
              int f64 = 0;
              const int what = repr::search_all(F, prj, mean, Y, iso, iso_ff, mean64, p, f64);
              const repr::Point64 pm = repr::mean_point_exact(pts[t], sz);
              double pe[3] = {pm.p[0], pm.p[1], pm.p[2]};
              repr::Stats st;
              repr::representative_exact(u, iso, c, t, pe, bx, st);
              // not found exactly where the reference goes on to its 26x26 retry
              if ((what == repr::kRedo) != (st.fail1 != 0) ||
                  (what == repr::kFound && (pe[0] != (double)p[0] || pe[1] != (double)p[1] || pe[2] != (double)p[2]))) {
                if (mism < 5) fprintf(stderr, "search: cell %d %d %d t %d (size %d, %d)\n", i, j, k, t, sz, what);
                mism++;
              }
              searched++;
            }
          }
          if (excl) {
            excluded++;
            continue;
          }
          float p[3] = {0, 0, 0};
          int prj = 0;
          float frame[repr::kFrameFloats];
          for (int q = 0; q < 8; q++) frame[q] = u[q];
          const int what = repr::vertex_point(repr::FrameCol{frame, 1}, em, sz, iso, ffx::ff_from_double(iso), (double)(float)iso == iso, p, prj);
          if (what == repr::kRedo) {
            redone++;
            continue;
          }
          if (what == repr::kW64) {
            p[2 - prj] = repr::vertex_w_f64(u, iso, p, prj);
            w64++;
          }
          const repr::Point64 pm = repr::mean_point_exact(pts[t], sz);
          double pe[3] = {pm.p[0], pm.p[1], pm.p[2]};
          repr::Stats st;
          repr::representative_exact(u, iso, c, t, pe, bx, st);
          if (st.fail1 || pe[0] != (double)p[0] || pe[1] != (double)p[1] || pe[2] != (double)p[2]) {
            if (mism < 5)
              fprintf(stderr, "cell %d %d %d t %d (size %d, %d): %.9g %.9g %.9g, not %.9g %.9g %.9g\n", i, j, k, t, sz,
                      what, p[0], p[1], p[2], pe[0], pe[1], pe[2]);
            mism++;
          }
        }
      }
  printf("%ld %ld %ld %ld %ld %ld\n", contours, mism, redone, w64, excluded, searched);
  return 0;
}

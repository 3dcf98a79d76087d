// Host driver for exciting_b200/csrc/sturm.cuh, used by tests/test_sturm_count.py.
//   sturm_harness in.txt
// in.txt lines:  minors n pivmin x d_0..d_n-1 e_0..e_n-2   -> the count, one per line on stdout
// (minors 1: leading minors, 0: quotients throughout, as the kernel takes them for large ||T||)
#include "sturm.cuh"

int main(int argc, char** argv) {
  FILE* in = argc == 2 ? fopen(argv[1], "r") : nullptr;
  if (!in) return 2;
  int minors, n;
  double pivmin, x;
  while (fscanf(in, "%d %d %lf %lf", &minors, &n, &pivmin, &x) == 4) {
    std::vector<double2> de(n);
    for (int i = 0; i < n; ++i)
      if (fscanf(in, "%lf", &de[i].x) != 1) return 4;
    de[0].y = 0.0;
    for (int i = 1; i < n; ++i) {
      double e;
      if (fscanf(in, "%lf", &e) != 1) return 4;
      de[i].y = e * e;
    }
    const double xs[NPT] = {x, x};
    int cnt[NPT];
    sturm_count(n, de.data(), xs, pivmin, minors != 0, cnt);
    printf("%d\n", cnt[1]);
  }
  fclose(in);
  return 0;
}

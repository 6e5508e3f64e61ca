// How many CTAs a decode product runs on.  Its (row group, 256-element block) units, `nb` per row group, are cut into one contiguous
// share per CTA; a row group that several CTAs share costs each of them a flush (partial sums, a counter) and the last one the sum.
#pragma once
#include <cstdint>

namespace gllmk {

// `ctas` resident CTAs (per_sm on an SM), several = more than one group of MMA columns, tiled = gemv.cu's kernel (gemv_raw.cu's
// otherwise).  With few units per CTA the shares differ by one
// unit in two or three, and a grid no larger than the longest share needs takes as many steps with fewer flushes — where its shares end
// at a row group's end.  Where they do not, or where the resident grid's do, the larger grid is the faster one: the rest of its CTAs
// leave their bandwidth to the others.  Time on the smaller grid over time on the larger one, one / five tokens, rows of nb blocks:
//   nb                                         4         8         12        14        16        20        28        32        43        56
//   longest share 4, 3 CTAs per SM (1400 units on 444)
//     Q4_K                                  .59/.74   .83/.90  1.05/1.11  .96/1.15  .88/1.04  .90/1.02  .93/1.03  .90/1.01  .95/1.08  .94/1.01
//     Q5_K                                  .79/.83   .93/.92  1.08/1.07 1.11/1.08  .97/.99  1.00/.98   .99/.98   .97/.97  1.05/1.08 1.03/.98
//   longest share 4, 2 CTAs per SM (952 on 296)
//     Q8_0                                  .72/.67   .81/.77  1.01/.98   .94/.95   .87/.88   .89/.87   .91/.86   .87/.85   .92/.94   .91/.85
//   longest share 3, 3 CTAs per SM (952 on 444)
//     Q4_K                                 1.13/1.30 1.13/1.34 1.00/1.10 1.06/1.24  .99/1.18 1.04/1.17 1.01/1.12 1.04/1.13  .99/1.05 1.01/1.09
//     Q5_K                                 1.25/1.21 1.27/1.26 1.09/1.07 1.24/1.16 1.18/1.15 1.17/1.14 1.14/1.12 1.16/1.11 1.10/1.02 1.11/1.07
//   longest share 3, 2 CTAs per SM (684 on 296)
//     Q8_0 x 1 / Q6_K x 5                  1.01/1.04 1.07/.97   .96/1.02  .97/1.02     -      .96/.99   .96/1.01  .98/.97   .97/.95   .95/.89
//   longest share 2 (512 on 444), five tokens
//     Q4_K / Q5_K                          1.07/1.12 1.06/1.07 1.02/1.02 1.00/1.00  .98/1.00  .99/.97   .95/.93   .92/.91   .98/.92   .85/.81
// (with one column group 1.0 - 1.14).  Five units and more: slower by up to 30 % but for eight that end at a row group's end.
inline int64_t decode_ctas(int64_t units, int64_t ctas, int per_sm, int64_t nb, bool several, bool tiled) {
    if (ctas > units) ctas = units;
    const int64_t longest = (units + ctas - 1) / ctas;
    bool fewer = false;
    if (longest == 4) fewer = nb % 12 != 0 && (per_sm < 3 || (nb % 4 == 0 && !(tiled && several && nb >= 16)));  // (shares of three and four both end at 12)
    else if (longest == 3) fewer = per_sm < 3 && nb >= 16 && units * 4 >= ctas * 9;
    else if (longest == 2) fewer = several && nb >= 16 && units * 10 >= ctas * 11;
    return fewer ? (units + longest - 1) / longest : ctas;
}

}  // namespace gllmk

// What the transfers compute from a particle's HessianData, built as host code, against the
// oracle's P and dP/dF: V0 P F^T (transfer_stress, transfer_stress2) and V0 dP F^T with dF = G F
// (hessian_stress with skew_system_inverse, hessian_stress2), and its product with G. Per family
// of singular values, "name value" pairs: the largest difference in units of the rounding
// unit of the type (2^-53, 2^-24) times the scale of the terms (below). A NaN is kept.
#include "mpm_math.cuh"
#include "mpm_oracle.h"
#include <cmath>
#include <cstdio>
#include <random>

using namespace mpm;

typedef long double Exact;      // the expected values, free of FP64 rounding
static void rotation(std::mt19937_64& g,Exact* R)
{
    std::normal_distribution<double> n(0.,1.);
    Exact w=n(g),x=n(g),y=n(g),z=n(g);
    const Exact s=1/std::sqrt(w*w+x*x+y*y+z*z);w*=s;x*=s;y*=s;z*=s;
    const Exact M[9]={1-2*(y*y+z*z),2*(x*y-w*z),2*(x*z+w*y),2*(x*y+w*z),1-2*(x*x+z*z),2*(y*z-w*x),2*(x*z-w*y),2*(y*z+w*x),1-2*(x*x+y*y)};
    for(int k=0;k<9;++k) R[k]=M[k];
}
static void worst(double& a,double b){if(!(b<=a)) a=b;}
static oracle::Mat<Exact,3> to_mat(const Exact* a){oracle::Mat<Exact,3> m;for(int k=0;k<9;++k) m.a[k/3][k%3]=a[k];return m;}

struct Particle {
    double F[9],R[9],G[9],lambda,mu,Je,V0;
    double A[9],B[9],bg,sA,sB,sbg;       // expected, and the scales of their terms
    HessianData<double> h;
    HessianData<float> hf;
};
static Particle particle(std::mt19937_64& g,int mode)
{
    std::uniform_real_distribution<double> u(-1.,1.);
    Particle p;
    Exact A[9],B[9],F[9],R[9];double s[3];
    rotation(g,A);rotation(g,B);
    for(double& x:s) x=mode==0?1+1e-3*u(g):mode==1?1+.2*u(g):mode==2?.3+.2*u(g):mode==3?2.5+1.5*u(g):1+.2*u(g);
    if(mode==4) s[2]=-(.3+.2*u(g));
    for(int i=0;i<3;++i) for(int j=0;j<3;++j){
        F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
        R[3*i+j]=A[3*i]*B[3*j]+A[3*i+1]*B[3*j+1]+A[3*i+2]*B[3*j+2];}
    for(int k=0;k<9;++k){p.F[k]=(double)F[k];p.R[k]=(double)R[k];}
    for(double& x:p.G) x=u(g);
    p.lambda=4e4*std::exp(2*u(g));p.mu=6e4*std::exp(2*u(g));p.V0=1e-6;
    oracle::Constitutive<Exact,3> cm;
    cm.Fe=to_mat(F);cm.Re=to_mat(R);cm.He=oracle::Cofactor(cm.Fe);cm.Je=(Exact)s[0]*s[1]*s[2];cm.lambda=p.lambda;cm.mu=p.mu;
    p.Je=(double)cm.Je;
    Exact G[9],dF[9];for(int k=0;k<9;++k) G[k]=p.G[k];
    mat_mul(G,F,dF);
    const oracle::Mat<Exact,3> P=cm.P(),dP=cm.Times_dP_dF(to_mat(dF));
    p.bg=0;
    for(int i=0;i<3;++i) for(int j=0;j<3;++j){
        Exact a=0,b=0;
        for(int k=0;k<3;++k){a+=P.a[i][k]*F[3*j+k];b+=dP.a[i][k]*F[3*j+k];}
        p.A[3*i+j]=p.V0*a;p.B[3*i+j]=p.V0*b;p.bg+=p.V0*b*p.G[3*i+j];}
    // E and S = I + E carry the rounding of numbers up to 1 + s; the rotation's 3x3 system
    // (eigenvalues s_i + s_j) magnifies that by at most (1 + s) over its least one
    double top=0,least=1e30;
    for(int i=0;i<3;++i){top=std::fmax(top,1+std::fabs(s[i]));least=std::fmin(least,std::fabs(s[i]+s[(i+1)%3]));}
    const double J=std::fabs(p.Je);
    p.sA=p.V0*(2*p.mu*top*top+p.lambda*J*(1+J));
    p.sB=3*p.V0*(2*p.mu*top*top*std::fmax(1.,top/least)+p.lambda*J*(1+J));   // |G_ij| <= 1, sums of three
    p.sbg=9*p.sB;
    hessian_data<double>(p.F,p.R,p.lambda,p.mu,p.Je,p.V0,p.h);
    float Ff[9],Rf[9];for(int k=0;k<9;++k){Ff[k]=(float)p.F[k];Rf[k]=(float)p.R[k];}
    hessian_data<float>(Ff,Rf,(float)p.lambda,(float)p.mu,(float)p.Je,(float)p.V0,p.hf);
    return p;
}
static const int ix[3][3]={{0,1,2},{1,3,4},{2,4,5}};

int main()
{
    const char* names[]={"light","strained","compressed","stretched","inverted"};
    for(int mode=0;mode<5;++mode){
        std::mt19937_64 g(3+mode);
        const double u64=std::ldexp(1.,-53),u32=std::ldexp(1.,-24);
        double A64=0,B64=0,A32=0,B32=0;
        for(int it=0;it<5000;++it){
            const Particle p[2]={particle(g,mode),particle(g,mode)};
            double A[6];transfer_stress<double>(p[0].h,false,A);
            const double* E=p[0].h.E;
            const double Sm[6]={1+E[0],E[1],E[2],1+E[3],E[4],1+E[5]};
            double Ki[6];skew_system_inverse(Sm,Ki);
            C3<double> G3[3],B3[3];double bg;
            for(int j=0;j<3;++j) G3[j]=c3<double>(p[0].G[j],p[0].G[3+j],p[0].G[6+j]);
            hessian_stress<double>(G3,Sm,p[0].h.c1,p[0].h.c2,p[0].h.c3,Ki,B3,bg);
            for(int i=0;i<3;++i) for(int j=0;j<3;++j){
                worst(A64,std::fabs(A[ix[i][j]]-p[0].A[3*i+j])/(u64*p[0].sA));
                const double b=i==0?B3[j].x:i==1?B3[j].y:B3[j].z;
                worst(B64,std::fabs(b-p[0].B[3*i+j])/(u64*p[0].sB));}
            worst(B64,std::fabs(bg-p[0].bg)/(u64*p[0].sbg));
            // FP32, two particles at once
            auto two=[&](auto f){return make_float2((float)f(p[0]),(float)f(p[1]));};
            float2 E2[6],S2[6],G2[3][3],A2[6],B2[3][3],bg2;
            for(int k=0;k<6;++k){
                E2[k]=two([&](const Particle& q){return q.hf.E[k];});
                S2[k]=k==0||k==3||k==5?padd(pdup(1.f),E2[k]):E2[k];}
            for(int k=0;k<9;++k) G2[k/3][k%3]=two([&](const Particle& q){return q.G[k];});
            const float2 c1=two([](const Particle& q){return q.hf.c1;}),c2=two([](const Particle& q){return q.hf.c2;}),c3=two([](const Particle& q){return q.hf.c3;});
            transfer_stress2(E2,c1,c3,A2);
            hessian_stress2(G2,S2,c1,c2,c3,B2,bg2);
            for(int h=0;h<2;++h){
                auto half=[&](float2 v){return (double)(h?v.y:v.x);};
                for(int i=0;i<3;++i) for(int j=0;j<3;++j){
                    worst(A32,std::fabs(half(A2[ix[i][j]])-p[h].A[3*i+j])/(u32*p[h].sA));
                    worst(B32,std::fabs(half(B2[i][j])-p[h].B[3*i+j])/(u32*p[h].sB));}
                worst(B32,std::fabs(half(bg2)-p[h].bg)/(u32*p[h].sbg));}}
        std::printf("%s_P64 %.4g %s_dP64 %.4g %s_P32 %.4g %s_dP32 %.4g ",names[mode],A64,names[mode],B64,names[mode],A32,names[mode],B32);}
    std::printf("\n");
    return 0;
}
